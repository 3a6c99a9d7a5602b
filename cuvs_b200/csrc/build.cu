// Index construction on the GPU: coarse k-means, rotation, PQ codebooks, encoding (extend),
// transform and the code unpack helper.
//
// What is kept from the reference (cpp/src/neighbors/ivf_pq/ivf_pq_build.cuh) is the data contract
// of the result, not the training procedure:
//   - trainset size rule .................. :1283-1290
//   - IP trains and predicts with L2 ....... :70-76
//   - rotation: identity when dim == rot_dim and not forced, else a random orthogonal matrix
//     (cpp/src/neighbors/ivf_pq/ivf_pq_build_common.cu:235-261)
//   - centers[l, dim] = |c_l|^2, zero tail; centers_rot = centers * R^T ........ :262-300
//   - codebooks stored [part, pq_len, book] with the book index fastest ........ :303-325
//   - encoding: residual = R (x - c_label); per subspace the codebook entry with the smallest
//     squared distance, lowest code on ties
//     (cpp/src/neighbors/ivf_pq/ivf_pq_process_and_fill_codes.cuh:84-126); codes written in the
//     interleaved layout (cpp/src/neighbors/ivf_pq/ivf_pq_codepacking.cuh:135-168)
// The coarse clustering is Lloyd k-means over all lists at once with the reference's balancing step
// between iterations (underfull clusters restart next to overfull ones, size-sorted donors,
// cpp/src/cluster/detail/kmeans_balanced.cuh:616-720) and re-seeding of empty clusters; the reference
// first clusters hierarchically (mesoclusters) to make training cheap, which the tensor-core
// labelling makes unnecessary here.  Unlike the reference's atomic slot allocation, vectors are placed
// in a list in input order, so extend is deterministic.
#include "ivf_pq.hpp"
#include "packed.cuh"
#include "search_internal.hpp"
#include "topk.cuh"

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <random>

namespace cuvs::neighbors::ivf_pq {

using namespace cuvs_b200;

namespace {

// ------------------------------------------------------------------------------------------------
// element conversion
// ------------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float to_float(T x);
template <> __device__ __forceinline__ float to_float<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_float<__half>(__half x) { return __half2float(x); }
template <> __device__ __forceinline__ float to_float<int8_t>(int8_t x) { return float(x) * (1.0f / 128.0f); }
template <> __device__ __forceinline__ float to_float<uint8_t>(uint8_t x) { return float(x) * (1.0f / 256.0f); }

// One warp per row: out[r, :dim] = mapping<float>(in[r * row_stride, :]) (optionally L2-normalised),
// out[r, dim] = pad, zero tail.
template <typename T>
__global__ void to_float_ext_kernel(const T* __restrict__ in, uint64_t n, uint64_t row_stride,
                                    uint32_t dim, uint32_t dim_ext, float pad, int normalize,
                                    float* __restrict__ out)
{
  const uint64_t r    = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (r >= n) { return; }
  const T* src = in + r * row_stride * dim;
  float* dst   = out + r * dim_ext;
  float inv    = 1.0f;
  if (normalize) {
    float ss = 0.0f;
    for (uint32_t i = lane; i < dim; i += 32) {
      float v = to_float<T>(src[i]);
      ss += v * v;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) { ss += __shfl_xor_sync(kFullMask, ss, d); }
    inv = ss > 0.0f ? 1.0f / sqrtf(ss) : 1.0f;
  }
  for (uint32_t i = lane; i < dim_ext; i += 32) {
    float v = 0.0f;
    if (i < dim) {
      v = to_float<T>(src[i]) * inv;
    } else if (i == dim) {
      v = pad;
    }
    dst[i] = v;
  }
}

void to_float_ext(raft::resources& res, const void* in, elem_t t, uint64_t n, uint64_t row_stride,
                  uint32_t dim, uint32_t dim_ext, float pad, bool normalize, float* out)
{
  if (n == 0) { return; }
  const unsigned blocks = unsigned(ceildiv<uint64_t>(n * 32, 256));
  switch (t) {
    case elem_t::f32:
      to_float_ext_kernel<float><<<blocks, 256, 0, res.stream>>>(static_cast<const float*>(in), n, row_stride, dim, dim_ext, pad, normalize, out);
      break;
    case elem_t::f16:
      to_float_ext_kernel<__half><<<blocks, 256, 0, res.stream>>>(static_cast<const __half*>(in), n, row_stride, dim, dim_ext, pad, normalize, out);
      break;
    case elem_t::i8:
      to_float_ext_kernel<int8_t><<<blocks, 256, 0, res.stream>>>(static_cast<const int8_t*>(in), n, row_stride, dim, dim_ext, pad, normalize, out);
      break;
    default:
      to_float_ext_kernel<uint8_t><<<blocks, 256, 0, res.stream>>>(static_cast<const uint8_t*>(in), n, row_stride, dim, dim_ext, pad, normalize, out);
  }
  CUDA_TRY(cudaGetLastError());
  res.launches++;
}

// ------------------------------------------------------------------------------------------------
// k-means update
// ------------------------------------------------------------------------------------------------
__global__ void accumulate_kernel(const float* __restrict__ x_ext, const uint32_t* __restrict__ labels,
                                  uint64_t n, uint32_t dim, uint32_t dim_ext, float* __restrict__ sums,
                                  uint32_t* __restrict__ counts)
{
  const uint64_t r    = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (r >= n) { return; }
  const uint32_t l = labels[r];
  const float* src = x_ext + r * dim_ext;
  float* dst       = sums + size_t(l) * dim;
  for (uint32_t i = lane; i < dim; i += 32) { atomicAdd(dst + i, src[i]); }
  if (lane == 0) { atomicAdd(counts + l, 1u); }
}

// One block per center: mean (or a re-seed from a pseudo-random row when the cluster is empty),
// squared norm into column `dim`, zero tail.
__global__ void finalize_centers_kernel(const float* __restrict__ sums, const uint32_t* __restrict__ counts,
                                        uint32_t dim, uint32_t dim_ext, const float* __restrict__ x_ext,
                                        uint64_t n, uint32_t seed, int normalize,
                                        float* __restrict__ centers)
{
  __shared__ float s_red[32];
  const uint32_t l   = blockIdx.x;
  const uint32_t cnt = counts[l];
  float* c           = centers + size_t(l) * dim_ext;
  const uint64_t rr  = (uint64_t(l) * 2654435761ull + uint64_t(seed) * 40503ull + 12345ull) % n;
  float ss           = 0.0f;
  for (uint32_t i = threadIdx.x; i < dim; i += blockDim.x) {
    float v = cnt > 0 ? sums[size_t(l) * dim + i] / float(cnt) : x_ext[rr * dim_ext + i];
    c[i]    = v;
    ss += v * v;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) { ss += __shfl_xor_sync(kFullMask, ss, d); }
  if ((threadIdx.x & 31) == 0) { s_red[threadIdx.x >> 5] = ss; }
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? s_red[threadIdx.x] : 0.0f;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) { v += __shfl_xor_sync(kFullMask, v, d); }
    if (threadIdx.x == 0) { s_red[0] = v; }
  }
  __syncthreads();
  float norm2 = s_red[0];
  if (normalize && norm2 > 0.0f) {
    const float inv = 1.0f / sqrtf(norm2);
    for (uint32_t i = threadIdx.x; i < dim; i += blockDim.x) { c[i] *= inv; }
    norm2 = 1.0f;
  }
  for (uint32_t i = dim + threadIdx.x; i < dim_ext; i += blockDim.x) { c[i] = i == dim ? norm2 : 0.0f; }
}

// centers_ext rows <- strided rows of x_ext (k-means initialisation)
__global__ void init_centers_kernel(const float* __restrict__ x_ext, uint64_t n, uint32_t n_lists,
                                    uint32_t dim_ext, float* __restrict__ centers)
{
  const uint32_t l = blockIdx.x;
  const uint64_t r = (uint64_t(l) * n) / n_lists;
  for (uint32_t i = threadIdx.x; i < dim_ext; i += blockDim.x) {
    centers[size_t(l) * dim_ext + i] = x_ext[r * dim_ext + i];
  }
}

// out[l, r] = sum_k R[r, k] * centers[l, k]
__global__ void rotate_centers_kernel(const float* __restrict__ centers, const float* __restrict__ rot,
                                      uint32_t n_lists, uint32_t dim, uint32_t dim_ext, uint32_t rot_dim,
                                      float* __restrict__ out)
{
  const uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (i >= uint64_t(n_lists) * rot_dim) { return; }
  const uint32_t l = uint32_t(i / rot_dim), r = uint32_t(i % rot_dim);
  const float* c = centers + size_t(l) * dim_ext;
  const float* R = rot + size_t(r) * dim;
  float acc      = 0.0f;
  for (uint32_t k = 0; k < dim; k++) { acc = __fmaf_rn(R[k], c[k], acc); }
  out[i] = acc;
}

// Balancing step of the coarse k-means (the reference's adjust_centers with size-sorted donors,
// cpp/src/cluster/detail/kmeans_balanced.cuh:520-720): one pseudo-random member row per cluster ...
__global__ void pick_member_kernel(const uint32_t* __restrict__ labels, uint64_t n, uint32_t seed,
                                   unsigned long long* __restrict__ member /* [n_lists], zeroed */)
{
  const uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (i >= n) { return; }
  // the row with the largest hash wins: a different member every iteration
  uint32_t h = uint32_t(i) * 2654435761u + seed * 40503u;
  h ^= h >> 15;
  h *= 2246822519u;
  h ^= h >> 13;
  atomicMax(member + labels[i], (static_cast<unsigned long long>(h) << 32) | uint32_t(i));
}

// ... and, per (receiver, donor) pair, the receiver's centre re-initialised next to the donor's centre,
// a small step (`offset`) towards one of the donor's rows, so that the next assignment splits the large
// cluster.  One block per pair; norm column and zero tail rewritten.
__global__ void adjust_centers_kernel(float* __restrict__ centers, const uint32_t* __restrict__ pairs /* [n_pairs][2] */,
                                      const unsigned long long* __restrict__ member,
                                      const float* __restrict__ x_ext, uint32_t dim, uint32_t dim_ext,
                                      float offset, int normalize)
{
  __shared__ float s_red[4];
  const uint32_t receiver = pairs[2 * blockIdx.x], donor = pairs[2 * blockIdx.x + 1];
  const uint64_t row      = member[donor] & 0xFFFFFFFFull;
  float* c                = centers + size_t(receiver) * dim_ext;
  const float* d          = centers + size_t(donor) * dim_ext;
  const float* x          = x_ext + row * dim_ext;
  float ss                = 0.0f;
  for (uint32_t i = threadIdx.x; i < dim; i += blockDim.x) {
    const float v = d[i] + offset * (x[i] - d[i]);
    c[i]          = v;
    ss += v * v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { ss += __shfl_xor_sync(kFullMask, ss, o); }
  if ((threadIdx.x & 31) == 0) { s_red[threadIdx.x >> 5] = ss; }
  __syncthreads();
  float norm2 = 0.0f;
  for (uint32_t w = 0; w < (blockDim.x >> 5); w++) { norm2 += s_red[w]; }
  if (normalize && norm2 > 0.0f) {
    const float inv = 1.0f / sqrtf(norm2);
    for (uint32_t i = threadIdx.x; i < dim; i += blockDim.x) { c[i] *= inv; }
    norm2 = 1.0f;
  }
  for (uint32_t i = dim + threadIdx.x; i < dim_ext; i += blockDim.x) { c[i] = i == dim ? norm2 : 0.0f; }
}

// Recompute column `dim` (squared norm) and the zero tail of padded centers in place.
__global__ void center_norms_kernel(float* __restrict__ centers, uint32_t n_lists, uint32_t dim,
                                    uint32_t dim_ext)
{
  const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= n_lists) { return; }
  float* c = centers + size_t(l) * dim_ext;
  float ss = 0.0f;
  for (uint32_t k = 0; k < dim; k++) { ss = __fmaf_rn(c[k], c[k], ss); }
  for (uint32_t k = dim; k < dim_ext; k++) { c[k] = k == dim ? ss : 0.0f; }
}

// Pad [n_lists, dim] centers to [n_lists, dim_ext] with the squared norm in column dim.
__global__ void pad_centers_kernel(const float* __restrict__ in, uint32_t n_lists, uint32_t dim,
                                   uint32_t dim_ext, float* __restrict__ out)
{
  const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= n_lists) { return; }
  float ss = 0.0f;
  for (uint32_t k = 0; k < dim; k++) {
    float v                       = in[size_t(l) * dim + k];
    out[size_t(l) * dim_ext + k] = v;
    ss                            = __fmaf_rn(v, v, ss);
  }
  for (uint32_t k = dim; k < dim_ext; k++) { out[size_t(l) * dim_ext + k] = k == dim ? ss : 0.0f; }
}

// ------------------------------------------------------------------------------------------------
// residuals
// ------------------------------------------------------------------------------------------------
// One block per selected row: out[i, :] = R * (x[rows[i]] - centers[label]) with each output
// accumulated in ascending k by FMA (identity rotation copies the difference).
__global__ void residual_kernel(const float* __restrict__ x_ext, const uint32_t* __restrict__ labels,
                                uint64_t row_stride, const float* __restrict__ centers,
                                const float* __restrict__ rot, int identity, uint32_t dim,
                                uint32_t dim_ext, uint32_t rot_dim, float* __restrict__ out)
{
  extern __shared__ float s_diff[];
  const uint64_t i   = blockIdx.x;
  const uint64_t row = i * row_stride;
  const float* x     = x_ext + row * dim_ext;
  const float* c     = centers + size_t(labels[row]) * dim_ext;
  for (uint32_t k = threadIdx.x; k < dim; k += blockDim.x) { s_diff[k] = __fsub_rn(x[k], c[k]); }
  __syncthreads();
  for (uint32_t r = threadIdx.x; r < rot_dim; r += blockDim.x) {
    float acc;
    if (identity) {
      acc = s_diff[r];
    } else {
      const float* R = rot + size_t(r) * dim;
      acc            = 0.0f;
      for (uint32_t k = 0; k < dim; k++) { acc = __fmaf_rn(R[k], s_diff[k], acc); }
    }
    out[i * rot_dim + r] = acc;
  }
}

// ------------------------------------------------------------------------------------------------
// PQ codebook training: one block per codebook, Lloyd iterations entirely in shared memory
// ------------------------------------------------------------------------------------------------
// Problem b trains `book` centers of `len` dims.
//   per_cluster == 0: b = subspace; points are slice b of every residual row (n_rows of them).
//   per_cluster == 1: b = list; points are all pq_dim slices of the residual rows
//                     row_ids[row_begin[b] .. row_begin[b+1]) (capped at max_rows).
__global__ void train_codebooks_kernel(const float* __restrict__ resid, uint32_t n_rows,
                                       uint32_t rot_dim, uint32_t pq_dim, uint32_t len, uint32_t book,
                                       int per_cluster, const uint32_t* __restrict__ row_ids,
                                       const uint32_t* __restrict__ row_begin, uint32_t max_rows,
                                       int n_iters, float* __restrict__ pq_centers)
{
  extern __shared__ float s_mem[];
  float* s_c       = s_mem;               // [book, len]
  float* s_sum     = s_c + book * len;    // [book, len]
  uint32_t* s_cnt  = reinterpret_cast<uint32_t*>(s_sum + book * len);  // [book]
  const uint32_t b = blockIdx.x;
  uint32_t rows0 = 0, nr = n_rows;
  if (per_cluster) {
    rows0 = row_begin[b];
    nr    = min(row_begin[b + 1] - rows0, max_rows);
  }
  const uint32_t n_pts = per_cluster ? nr * pq_dim : nr;
  float* out           = pq_centers + size_t(b) * len * book;
  if (n_pts == 0) {
    for (uint32_t i = threadIdx.x; i < len * book; i += blockDim.x) { out[i] = 0.0f; }
    return;
  }
  auto point = [&](uint32_t p) -> const float* {
    if (per_cluster) {
      const uint32_t row = row_ids[rows0 + p / pq_dim];
      return resid + size_t(row) * rot_dim + (p % pq_dim) * len;
    }
    return resid + size_t(p) * rot_dim + b * len;
  };
  // init: evenly strided points
  for (uint32_t i = threadIdx.x; i < book * len; i += blockDim.x) {
    const uint32_t c = i / len, k = i % len;
    s_c[i]           = point(uint32_t((uint64_t(c) * n_pts) / book))[k];
  }
  __syncthreads();
  for (int it = 0; it < n_iters; it++) {
    for (uint32_t i = threadIdx.x; i < book * len; i += blockDim.x) { s_sum[i] = 0.0f; }
    for (uint32_t i = threadIdx.x; i < book; i += blockDim.x) { s_cnt[i] = 0; }
    __syncthreads();
    for (uint32_t p = threadIdx.x; p < n_pts; p += blockDim.x) {
      const float* x = point(p);
      float best     = INFINITY;
      uint32_t bc    = 0;
      for (uint32_t c = 0; c < book; c++) {
        float d2 = 0.0f;
        for (uint32_t k = 0; k < len; k++) {
          float t = x[k] - s_c[c * len + k];
          d2 += t * t;
        }
        if (d2 < best) {
          best = d2;
          bc   = c;
        }
      }
      for (uint32_t k = 0; k < len; k++) { atomicAdd(&s_sum[bc * len + k], x[k]); }
      atomicAdd(&s_cnt[bc], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < book * len; i += blockDim.x) {
      const uint32_t c = i / len, k = i % len;
      if (s_cnt[c] > 0) {
        s_c[i] = s_sum[i] / float(s_cnt[c]);
      } else {
        // empty: re-seed from a pseudo-random point, nudged so that duplicates separate
        const uint32_t p = uint32_t((uint64_t(c) * 2654435761ull + uint64_t(it + 1) * 97003ull) % n_pts);
        s_c[i]           = point(p)[k] * (1.0f + 1e-3f * float((c % 7) + 1));
      }
    }
    __syncthreads();
  }
  // stored transposed: [len, book]
  for (uint32_t i = threadIdx.x; i < book * len; i += blockDim.x) {
    const uint32_t c = i / len, k = i % len;
    out[size_t(k) * book + c] = s_c[i];
  }
}

// ------------------------------------------------------------------------------------------------
// encoder
// ------------------------------------------------------------------------------------------------

// Differences of the rows (taken in `order`) to the centres of their lists.  One thread per component.
__global__ void difference_kernel(const float* __restrict__ x_ext, const uint32_t* __restrict__ labels,
                                  const uint32_t* __restrict__ order, const float* __restrict__ centers, uint32_t n, uint32_t dim,
                                  uint32_t dim_ext, float* __restrict__ out)
{
  const uint64_t t = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (t >= uint64_t(n) * dim) { return; }
  const uint32_t i = uint32_t(t / dim), k = uint32_t(t - uint64_t(i) * dim);
  const uint32_t row = order ? order[i] : i;
  out[t] = __fsub_rn(x_ext[size_t(row) * dim_ext + k], centers[size_t(labels[row]) * dim_ext + k]);
}

// Codes of per-subspace codebooks, one byte each: codes[i * out_stride + j] = the codeword of subspace j with the smallest
// squared distance (a fused multiply-add chain over its components), lowest code on ties.  Vector i is row order[i]
// of x, minus the centre of its list where `centers` is given.
// What bounds it: the FMA pipe, at four operations per vector and codeword of two components.  Thread = four vectors, so that a
// codeword read from shared memory (broadcast) serves four; two codewords per instruction (fp32x2); the minimum of
// eight distances is compared with the best so far, and only the winning eight are looked at one by one.
// One warp per vector with the codebook read through L1 took 24.8 ms for 1 M rows of 48 x 8 bits.
// kLen: components per subspace, 0 = any number.
constexpr uint32_t kEncVecs = 4;
template <uint32_t kLen>
__host__ __device__ constexpr uint32_t enc_subspaces() { return kLen == 0 || kLen > 4 ? 1u : (kLen > 2 ? 2u : 4u); }
template <uint32_t kLen>
__global__ void __launch_bounds__(256)
encode_subspaces_kernel(const float* __restrict__ x, uint32_t x_stride, const uint32_t* __restrict__ order,
                        const uint32_t* __restrict__ labels, const float* __restrict__ centers, uint32_t c_stride, uint32_t n,
                        const float* __restrict__ pq_centers, uint32_t pq_dim, uint32_t len_rt, uint32_t book, int in_smem,
                        uint8_t* __restrict__ codes, uint32_t out_stride)
{
  extern __shared__ __align__(16) float s_book[];
  constexpr uint32_t kSub = enc_subspaces<kLen>();
  constexpr uint32_t kEnt = kLen == 0 || kLen > 4 ? 4u : 8u;  // codewords per step
  const uint32_t len = kLen > 0 ? kLen : len_rt;
  const uint32_t j0 = blockIdx.y * kSub, nj = min(kSub, pq_dim - j0);
  if (in_smem) {
    const float4* src = reinterpret_cast<const float4*>(pq_centers + size_t(j0) * len * book);
    float4* dst       = reinterpret_cast<float4*>(s_book);
    for (uint32_t i = threadIdx.x; i < nj * len * book / 4; i += 256) { dst[i] = __ldg(src + i); }
    __syncthreads();
  }
  const float* book0 = in_smem ? s_book : pq_centers + size_t(j0) * len * book;
  const float* xr[kEncVecs];
  const float* cr[kEncVecs];
  uint32_t code[kEncVecs];
  const uint32_t i0 = blockIdx.x * (256u * kEncVecs) + threadIdx.x;
#pragma unroll
  for (uint32_t v = 0; v < kEncVecs; v++) {
    const uint32_t i   = min(i0 + v * 256u, n - 1u);
    const uint32_t row = order ? order[i] : i;
    xr[v]              = x + size_t(row) * x_stride + j0 * len;
    cr[v]              = centers ? centers + size_t(labels[row]) * c_stride + j0 * len : nullptr;
    code[v]            = 0u;
  }
  auto component = [&](uint32_t v, uint32_t k) {
    const float a = __ldg(xr[v] + k);
    return centers ? __fsub_rn(a, __ldg(cr[v] + k)) : a;
  };
  // the first of kEnt codewords at `b` whose distance is the smallest one found
  auto pick = [&](const float* b, float best, auto&& comp) {
    uint32_t first = 0;
    for (int e = int(kEnt) - 1; e >= 0; e--) {
      float d2 = 0.0f;
      for (uint32_t k = 0; k < len; k++) {
        const float t = __fsub_rn(comp(k), b[size_t(k) * book + e]);
        d2            = __fmaf_rn(t, t, d2);
      }
      if (d2 == best) { first = uint32_t(e); }
    }
    return first;
  };
#pragma unroll
  for (uint32_t s = 0; s < kSub; s++) {
    if (s >= nj) { break; }
    const float* bk = book0 + size_t(s) * len * book;
    float best[kEncVecs];
    uint32_t at[kEncVecs];
#pragma unroll
    for (uint32_t v = 0; v < kEncVecs; v++) {
      best[v] = INFINITY;
      at[v]   = 0u;
    }
    auto reduce = [&](uint32_t v, const uint64_t (&d)[kEnt / 2], uint32_t b0) {
      float m = min3(lo2(d[0]), hi2(d[0]), fminf(lo2(d[1]), hi2(d[1])));
      if constexpr (kEnt == 8) {
        m = min3(m, lo2(d[2]), hi2(d[2]));
        m = min3(m, lo2(d[3]), hi2(d[3]));
      }
      if (m < best[v]) {
        best[v] = m;
        at[v]   = b0;
      }
    };
    if constexpr (kLen > 0) {
      float r[kEncVecs][kLen];
#pragma unroll
      for (uint32_t v = 0; v < kEncVecs; v++) {
#pragma unroll
        for (uint32_t k = 0; k < kLen; k++) { r[v][k] = component(v, s * kLen + k); }
      }
#pragma unroll 1
      for (uint32_t b0 = 0; b0 < book; b0 += kEnt) {
        uint64_t c[kLen][kEnt / 2];
#pragma unroll
        for (uint32_t k = 0; k < kLen; k++) {
#pragma unroll
          for (uint32_t e = 0; e < kEnt / 4; e++) {
            const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(bk + k * book + b0 + 4 * e);
            c[k][2 * e]        = y.x;
            c[k][2 * e + 1]    = y.y;
          }
        }
#pragma unroll
        for (uint32_t v = 0; v < kEncVecs; v++) {
          uint64_t d[kEnt / 2];
#pragma unroll
          for (uint32_t k = 0; k < kLen; k++) {
            const uint64_t rr = dup2(r[v][k]);
#pragma unroll
            for (uint32_t e = 0; e < kEnt / 2; e++) {
              const uint64_t t = sub2(rr, c[k][e]);
              d[e]             = k == 0 ? mul2(t, t) : fma2(t, t, d[e]);  // the chain starts from +0
            }
          }
          reduce(v, d, b0);
        }
      }
#pragma unroll
      for (uint32_t v = 0; v < kEncVecs; v++) {
        // (no finite distance at all: code 0)
        if (best[v] < INFINITY) {
          uint32_t first = 0;
#pragma unroll
          for (int e = int(kEnt) - 1; e >= 0; e--) {
            float d2 = 0.0f;
#pragma unroll
            for (uint32_t k = 0; k < kLen; k++) {
              const float t = __fsub_rn(r[v][k], bk[k * book + at[v] + e]);
              d2            = __fmaf_rn(t, t, d2);
            }
            if (d2 == best[v]) { first = uint32_t(e); }
          }
          code[v] |= (at[v] + first) << (8u * s);
        }
      }
    } else {
      for (uint32_t b0 = 0; b0 < book; b0 += kEnt) {
        uint64_t d[kEncVecs][kEnt / 2];
#pragma unroll
        for (uint32_t v = 0; v < kEncVecs; v++) { d[v][0] = d[v][1] = 0ull; }
        for (uint32_t k = 0; k < len; k++) {
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(bk + size_t(k) * book + b0);
#pragma unroll
          for (uint32_t v = 0; v < kEncVecs; v++) {
            const uint64_t rr = dup2(component(v, k));
            const uint64_t t0 = sub2(rr, y.x), t1 = sub2(rr, y.y);
            d[v][0] = fma2(t0, t0, d[v][0]);
            d[v][1] = fma2(t1, t1, d[v][1]);
          }
        }
#pragma unroll
        for (uint32_t v = 0; v < kEncVecs; v++) { reduce(v, d[v], b0); }
      }
#pragma unroll
      for (uint32_t v = 0; v < kEncVecs; v++) {
        if (best[v] < INFINITY) { code[v] = at[v] + pick(bk + at[v], best[v], [&](uint32_t k) { return component(v, k); }); }
      }
    }
  }
#pragma unroll
  for (uint32_t v = 0; v < kEncVecs; v++) {
    const uint32_t i = i0 + v * 256u;
    if (i >= n) { continue; }
    uint8_t* o = codes + size_t(i) * out_stride + j0;
    if (kSub == 4 && nj == 4 && (reinterpret_cast<uintptr_t>(o) & 3u) == 0) {
      *reinterpret_cast<uint32_t*>(o) = code[v];
    } else {
      for (uint32_t s = 0; s < nj; s++) { o[s] = uint8_t(code[v] >> (8u * s)); }
    }
  }
}

// The same codes through a table of cells, for codewords of at most four components and many vectors: the space around a
// subspace's codewords is cut into kCells cells, and a cell names the codewords that can be the nearest one of a point in it,
// so that a vector looks at those instead of all of them: of 256 codewords some 2 with one or two components, 5 with three,
// 12 with four (k-means codebooks of normal and of heavy-tailed residuals).
//
// An axis is cut evenly in u = z / sqrt(1 + z^2), z the distance to the mean codeword in units of twice the mean deviation: fine
// cells where codewords are dense (even cuts of the axis itself: 6 codewords instead of 2 on heavy tails).
//
// A codeword c is left out of a cell where some other c' is nearer at every point of it by more than rounding can hide:
// |x - c'|^2 - |x - c|^2 is linear in x, so its maximum over the cell (a little enlarged: the cell of a point is found with
// rounding) is that of a corner.  What is left always holds the codeword that the comparison of all distances finds, and
// is compared in the same order with the same arithmetic; points far outside, NaN among them, are compared with all.
constexpr uint32_t kCells = 4096, kCellSpill = 16384;
template <uint32_t kLen>
struct cell_shape {
  static constexpr uint32_t axis  = kLen == 1 ? 4096u : (kLen == 2 ? 64u : (kLen == 3 ? 16u : 8u));
  static constexpr uint32_t bytes = kLen <= 2 ? 8u : 16u;   // of a cell
  static constexpr uint32_t codes = bytes - 1u;             // that fit it
  static constexpr uint32_t subs  = kLen <= 2 ? 4u : 2u;    // subspaces of a block of the encoder
  static constexpr uint32_t sure  = kLen <= 2 ? 3u : (kLen == 3 ? 4u : 8u);  // codewords looked at without asking how many there are
  // cells of a warp along axis k, and warps of a patch of 256 cells
  static __host__ __device__ constexpr uint32_t lanes(uint32_t k)
  {
    return kLen == 1 ? 32u : (kLen == 2 ? (k == 0 ? 8u : 4u) : (kLen == 3 ? (k == 2 ? 2u : 4u) : (k == 0 ? 4u : 2u)));
  }
  static __host__ __device__ constexpr uint32_t warps(uint32_t k) { return kLen == 1 ? 8u : (kLen == 2 ? (k == 0 ? 2u : 4u) : (kLen == 4 && k == 0 ? 1u : 2u)); }
};
// A table: cells, then the codes of long cells.  A cell: count, codes (unused places repeat the last one); count kCellLong:
// {-, codes (byte 1), -, offset of them in `spill` (bytes 4-7)}; kCellAll: every codeword.  frame: per component {mean, 1 / deviation,
// low end in u, cells per u}, ends: {lowest, highest} value that the edge cells hold.
constexpr uint32_t kCellLong = 0xFEu, kCellAll = 0xFFu;
template <uint32_t kLen>
struct code_table {
  uint4 cell[kCells * cell_shape<kLen>::bytes / 16];
  uint8_t spill[kCellSpill];
  float4 frame[kLen];
  float2 ends[4];
  uint32_t n_spill, pad[3];
};

// Block: a patch of 256 cells of subspace blockIdx.x.  The codewords that can matter are found for the patch, of those the ones
// for a warp's 32 cells, of those the ones for a cell.  What bounds it: the instructions of the comparisons (from the whole
// codebook for every cell: 119 us instead of 43 for 64 subspaces of two components and 256 codewords).
template <uint32_t kLen>
__global__ void __launch_bounds__(256)
code_cells_kernel(const float* __restrict__ pq_centers, uint32_t book, code_table<kLen>* __restrict__ tables)
{
  using shape = cell_shape<kLen>;
  constexpr uint32_t kAxis = shape::axis, kShort = 64;
  __shared__ float s_c[kLen][256];
  constexpr uint32_t kFirst = kLen <= 2 ? 4u : 16u;  // codewords nearest to a warp's middle that the others are compared with
  __shared__ uint8_t s_left[256], s_near[8][256], s_first[8][kFirst];  // codewords that matter to the patch, to a warp: ascending
  __shared__ uint8_t s_kept[256][kShort + 4];
  __shared__ float s_red[3][8];
  __shared__ unsigned long long s_mid[8];
  __shared__ uint32_t s_warp[8];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  auto& t = tables[blockIdx.x];
  for (uint32_t i = tid; i < kLen * book; i += 256) { s_c[i / book][i % book] = pq_centers[size_t(blockIdx.x) * kLen * book + i]; }
  __syncthreads();
  auto block_reduce = [&](float a, float b, float c, float& mn, float& mx, float& sum) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a = fminf(a, __shfl_xor_sync(kFullMask, a, o));
      b = fmaxf(b, __shfl_xor_sync(kFullMask, b, o));
      c += __shfl_xor_sync(kFullMask, c, o);
    }
    if (lane == 0) {
      s_red[0][warp] = a;
      s_red[1][warp] = b;
      s_red[2][warp] = c;
    }
    __syncthreads();
    mn = s_red[0][0]; mx = s_red[1][0]; sum = s_red[2][0];
    for (uint32_t w = 1; w < 8; w++) {
      mn = fminf(mn, s_red[0][w]);
      mx = fmaxf(mx, s_red[1][w]);
      sum += s_red[2][w];
    }
    __syncthreads();
  };
  float lo[kLen], hi[kLen], mean[kLen], dev[kLen], range = 0.0f;
  bool usable = true;
#pragma unroll
  for (uint32_t k = 0; k < kLen; k++) {
    const float v = s_c[k][min(tid, book - 1u)], in = tid < book ? 1.0f : 0.0f;
    float x0, x1, sum;
    block_reduce(v, v, v * in, lo[k], hi[k], sum);
    mean[k] = sum / float(book);
    block_reduce(v, v, fabsf(v - mean[k]) * in, x0, x1, sum);
    dev[k] = 2.0f * sum / float(book);
    range  = fmaxf(range, hi[k] - lo[k]);
    usable = __syncthreads_and(fabsf(v) < 1e12f) && usable;  // (false for NaN)
  }
  // (all codewords equal: the first one wins everywhere)
  const bool alone = usable && range == 0.0f;
  // (squares of a box this small or large would leave fp32)
  usable = usable && range > 1e-12f;
  constexpr float kFarOut = kLen <= 2 ? 1.0f : 0.25f;  // (edge cells that reach farther name more codewords)
  float u0[kLen], du[kLen], end0[kLen], end1[kLen];  // low end and width of the cells in u, ends of the edge cells
#pragma unroll
  for (uint32_t k = 0; k < kLen; k++) {
    dev[k]        = fmaxf(dev[k], 0.01f * range);
    const float r = fmaxf(hi[k] - lo[k], 0.01f * range);
    const float z0 = (lo[k] - 0.25f * r - mean[k]) / dev[k], z1 = (hi[k] + 0.25f * r - mean[k]) / dev[k];
    u0[k]   = z0 * rsqrtf(1.0f + z0 * z0);
    du[k]   = (z1 * rsqrtf(1.0f + z1 * z1) - u0[k]) / float(kAxis);
    end0[k] = lo[k] - 0.25f * r - kFarOut * range;
    end1[k] = hi[k] + 0.25f * r + kFarOut * range;
    // (the ends of a cell are off by rounding of their own size: 1/64 of its width has to cover that)
    usable = usable && dev[k] * du[k] > 1.6e-5f * fmaxf(fabsf(lo[k]), fabsf(hi[k]));
    if (blockIdx.y == 0 && tid == 0) {
      t.frame[k] = make_float4(mean[k], 1.0f / dev[k], u0[k], 1.0f / du[k]);
    }
  }
  if (blockIdx.y == 0 && tid == 0) {
    // (not usable: nothing lies between the ends)
#pragma unroll
    for (uint32_t k = 0; k < kLen; k++) {
      t.ends[k] = usable ? make_float2(end0[k], end1[k]) : (alone ? make_float2(-INFINITY, INFINITY) : make_float2(INFINITY, -INFINITY));
    }
  }
  // value at cell position p of axis k
  auto at = [&](uint32_t k, float p) {
    const float u = fminf(fmaxf(u0[k] + p * du[k], -0.9999999f), 0.9999999f);
    return mean[k] + dev[k] * u * rsqrtf(1.0f - u * u);
  };
  // ends of cells i .. i + n of axis k, enlarged by 1/64 of a cell (a point's cell position is off by less than 2^-8)
  auto span = [&](uint32_t k, uint32_t i, uint32_t n, float& a, float& b) {
    a = i == 0 ? end0[k] : at(k, float(i) - 0.015625f);
    b = i + n == kAxis ? end1[k] : at(k, float(i + n) + 0.015625f);
  };
  // `far`: no point of the box is farther from a codeword (squared); rounding of two distances and of the difference below is
  // at most 20 roundings of 2^-24 of it
  auto far_of = [&](const float (&a)[kLen], const float (&b)[kLen]) {
    float far = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < kLen; k++) {
      const float d = fmaxf(b[k] - lo[k], hi[k] - a[k]);
      far           = __fmaf_rn(d, d, far);
    }
    return far;
  };
  // codeword p is nearer than e in all of the box
  auto beats = [&](uint32_t p, uint32_t e, const float (&a)[kLen], const float (&b)[kLen], float margin) {
    float g = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < kLen; k++) {
      const float cp = s_c[k][p], ce = s_c[k][e], d = cp - ce;
      g += fmaxf(d * ((cp - a[k]) + (ce - a[k])), d * ((cp - b[k]) + (ce - b[k])));
    }
    return g < -margin;
  };
  auto to_middle = [&](uint32_t e, const float (&a)[kLen], const float (&b)[kLen]) {
    float d2 = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < kLen; k++) {
      const float d = 0.5f * (a[k] + b[k]) - s_c[k][e];
      d2            = __fmaf_rn(d, d, d2);
    }
    return d2;
  };
  // this thread's cell, its warp's and the block's
  uint32_t cell = 0, stride = 1, patch = blockIdx.y, in_lane = lane, in_warp = warp;
  float a[kLen], b[kLen], wa[kLen], wb[kLen], pa[kLen], pb[kLen];
#pragma unroll
  for (uint32_t k = 0; k < kLen; k++) {
    const uint32_t nl = shape::lanes(k), nw = shape::warps(k), np = kAxis / (nl * nw);
    const uint32_t p0 = (patch % np) * nl * nw, w0 = p0 + (in_warp % nw) * nl, i = w0 + in_lane % nl;
    patch /= np;
    in_warp /= nw;
    in_lane /= nl;
    cell += i * stride;
    stride *= kAxis;
    span(k, i, 1, a[k], b[k]);
    span(k, w0, nl, wa[k], wb[k]);
    span(k, p0, nl * nw, pa[k], pb[k]);
  }
  // e is beaten by one of the n codewords of `list` in the box, or equals one of lower code (which wins every tie)
  auto beaten_by = [&](const uint8_t* list, uint32_t n, uint32_t e, const float (&a)[kLen], const float (&b)[kLen], float margin) {
    for (uint32_t o = 0; o < n; o++) {
      const uint32_t p = list[o];
      bool same        = p < e;
#pragma unroll
      for (uint32_t k = 0; k < kLen; k++) { same = same && s_c[k][p] == s_c[k][e]; }
      if (same || beats(p, e, a, b, margin)) { return true; }
    }
    return false;
  };
  uint32_t n_near = 0;
  if (usable) {
    // the patch: what the one nearest to its middle leaves
    auto nearest = [&](uint64_t key) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const uint64_t other = shfl_u64(key, int(lane) ^ o);
        key                  = other < key ? other : key;
      }
      return key;
    };
    auto key_of = [&](uint32_t e, const float (&a)[kLen], const float (&b)[kLen]) {
      return (uint64_t(__float_as_uint(to_middle(e, a, b))) << 32) | e;
    };
    uint64_t key = nearest(tid < book ? key_of(tid, pa, pb) : ~0ull);
    if (lane == 0) { s_mid[warp] = key; }
    __syncthreads();
    for (uint32_t w = 0; w < 8; w++) { key = s_mid[w] < key ? s_mid[w] : key; }
    const bool stays = tid < book && !beats(uint32_t(key), tid, pa, pb, far_of(pa, pb) * 4e-6f);
    const unsigned m = __ballot_sync(kFullMask, stays);
    if (lane == 0) { s_warp[warp] = __popc(m); }
    __syncthreads();
    uint32_t at = 0, n_left = 0;
    for (uint32_t w = 0; w < 8; w++) {
      if (w < warp) { at += s_warp[w]; }
      n_left += s_warp[w];
    }
    if (stays) { s_left[at + __popc(m & ((1u << lane) - 1u))] = uint8_t(tid); }
    __syncthreads();
    // the warp: what the kFirst nearest to its middle leave
    uint64_t keys[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) { keys[i] = i * 32u + lane < n_left ? key_of(s_left[i * 32u + lane], wa, wb) : ~0ull; }
    const uint32_t n_first = min(kFirst, n_left);
    for (uint32_t f = 0; f < n_first; f++) {
      uint64_t mine = keys[0];
#pragma unroll
      for (uint32_t i = 1; i < 8; i++) { mine = keys[i] < mine ? keys[i] : mine; }
      const uint64_t first = nearest(mine);
#pragma unroll
      for (uint32_t i = 0; i < 8; i++) { keys[i] = keys[i] == first ? ~0ull : keys[i]; }
      if (lane == 0) { s_first[warp][f] = uint8_t(first); }
    }
    __syncwarp();
    const float w_margin = far_of(wa, wb) * 4e-6f;
    for (uint32_t i0 = 0; i0 < n_left; i0 += 32) {
      const uint32_t c    = i0 + lane < n_left ? s_left[i0 + lane] : 0u;
      const bool in       = i0 + lane < n_left && !beaten_by(s_first[warp], n_first, c, wa, wb, w_margin);
      const unsigned in_m = __ballot_sync(kFullMask, in);
      if (in) { s_near[warp][n_near + __popc(in_m & ((1u << lane) - 1u))] = uint8_t(c); }
      n_near += __popc(in_m);
    }
    __syncwarp();
  }
  uint32_t n = 0xFFFFu;
  if (alone) {
    n              = 1;
    s_kept[tid][0] = 0;
  }
  if (usable) {
    // the cell
    const float margin = far_of(a, b) * 4e-6f;
    uint32_t mid = 0;
    float best   = INFINITY;
    for (uint32_t i = 0; i < n_near; i++) {
      const float d2 = to_middle(s_near[warp][i], a, b);
      if (d2 < best) {
        best = d2;
        mid  = s_near[warp][i];
      }
    }
    // (most are beaten by the one nearest to the middle, nearly all others by one already kept)
    n = 0;
    for (uint32_t i = 0; i < n_near && n <= kShort; i++) {
      const uint32_t e = s_near[warp][i];
      if (!beats(mid, e, a, b, margin) && !beaten_by(s_kept[tid], n, e, a, b, margin)) {
        if (n < kShort) { s_kept[tid][n] = uint8_t(e); }
        n++;
      }
    }
    if (n <= kShort) {
      // without those that one kept after them beats
      uint32_t m = 0;
      for (uint32_t i = 0; i < n; i++) {
        const uint32_t e = s_kept[tid][i];
        if (!beaten_by(s_kept[tid] + i + 1, n - i - 1, e, a, b, margin)) { s_kept[tid][m++] = uint8_t(e); }
      }
      n = m;
    }
  }
  uint32_t w[shape::bytes / 4] = {kCellAll};
  if (n <= shape::codes) {
    w[0] = n;
#pragma unroll
    for (uint32_t i = 0; i < shape::codes; i++) { w[(i + 1) / 4] |= uint32_t(s_kept[tid][min(i, n - 1u)]) << (((i + 1) & 3u) * 8u); }
  } else if (n <= kShort) {
    const uint32_t from = atomicAdd(&t.n_spill, n);
    if (from + n <= kCellSpill) {
      for (uint32_t i = 0; i < n; i++) { t.spill[from + i] = s_kept[tid][i]; }
      w[0] = kCellLong | (n << 8);
      w[1] = from;
    }
  }
  auto* out = reinterpret_cast<uint32_t*>(t.cell) + cell * (shape::bytes / 4);
#pragma unroll
  for (uint32_t i = 0; i < shape::bytes / 4; i++) { out[i] = w[i]; }
}

// Block: the tables of a few subspaces in shared memory, `rows_per_block` vectors, a thread per vector.  What bounds it: the
// instructions and shared-memory wavefronts of the look-ups (a cell, then the components of a few codewords, each at random
// places).  1,000,003 rows of 48 x 2 components, 256 codewords: 2,180 us by comparing all, 361 us so.
template <uint32_t kLen>
__global__ void __launch_bounds__(1024, 1)
encode_cells_kernel(const float* __restrict__ x, uint32_t x_stride, const uint32_t* __restrict__ order,
                    const uint32_t* __restrict__ labels, const float* __restrict__ centers, uint32_t c_stride, uint32_t n,
                    const float* __restrict__ pq_centers, const code_table<kLen>* __restrict__ tables, uint32_t pq_dim,
                    uint32_t book, uint32_t rows_per_block, int vec, uint8_t* __restrict__ codes)
{
  using shape = cell_shape<kLen>;
  constexpr uint32_t kSub = shape::subs, kN = kSub * kLen, kAxis = shape::axis, kWords = shape::bytes / 4;
  extern __shared__ __align__(16) uint8_t s_tables[];
  auto* s_book = reinterpret_cast<float*>(s_tables + size_t(kSub) * kCells * shape::bytes);  // [kSub][book][kLen]
  const uint32_t tid = threadIdx.x;
  const uint32_t j0 = blockIdx.x * kSub, nj = min(kSub, pq_dim - j0);
  constexpr uint32_t kPer = kCells * shape::bytes / 16;
  for (uint32_t i = tid; i < nj * kPer; i += 1024u) { reinterpret_cast<uint4*>(s_tables)[i] = __ldg(tables[j0 + i / kPer].cell + i % kPer); }
  for (uint32_t i = tid; i < nj * kLen * book; i += 1024u) {
    const uint32_t s = i / (kLen * book), k = i / book % kLen, e = i % book;
    s_book[(s * book + e) * kLen + k] = __ldg(pq_centers + size_t(j0) * kLen * book + i);
  }
  __shared__ float4 s_frame[kN];
  __shared__ float2 s_ends[kN];
  if (tid < nj * kLen) {
    s_frame[tid] = __ldg(&tables[j0 + tid / kLen].frame[tid % kLen]);
    s_ends[tid]  = __ldg(&tables[j0 + tid / kLen].ends[tid % kLen]);
  }
  __syncthreads();
  const uint32_t end = min(n, (blockIdx.y + 1u) * rows_per_block);
  for (uint32_t i = blockIdx.y * rows_per_block + tid; i < end; i += 1024u) {
    const uint32_t row = order ? __ldg(order + i) : i;
    const float* xr    = x + size_t(row) * x_stride + j0 * kLen;
    const float* cr    = centers ? centers + size_t(__ldg(labels + row)) * c_stride + j0 * kLen : nullptr;
    float r[kN];
    if (kN % 4 == 0 && vec && nj == kSub) {
#pragma unroll
      for (uint32_t v = 0; v + 4 <= kN; v += 4) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(xr + v));
        r[v] = q.x; r[v + 1] = q.y; r[v + 2] = q.z; r[v + 3] = q.w;
      }
      if (centers) {
#pragma unroll
        for (uint32_t v = 0; v + 4 <= kN; v += 4) {
          const float4 c = __ldg(reinterpret_cast<const float4*>(cr + v));
          r[v] = __fsub_rn(r[v], c.x); r[v + 1] = __fsub_rn(r[v + 1], c.y);
          r[v + 2] = __fsub_rn(r[v + 2], c.z); r[v + 3] = __fsub_rn(r[v + 3], c.w);
        }
      }
    } else {
#pragma unroll
      for (uint32_t v = 0; v < kN; v++) {
        r[v] = v < nj * kLen ? __ldg(xr + v) : 0.0f;
        if (centers && v < nj * kLen) { r[v] = __fsub_rn(r[v], __ldg(cr + v)); }
      }
    }
    uint32_t cell[kSub][kWords], from[kSub], code[kSub];
    float best[kSub];
    auto look = [&](uint32_t s, uint32_t e) {
      const float* c = s_book + (s * book + e) * kLen;
      float y[kLen];
      if constexpr (kLen == 2) {
        const float2 v = *reinterpret_cast<const float2*>(c);
        y[0] = v.x; y[1] = v.y;
      } else if constexpr (kLen == 4) {
        const float4 v = *reinterpret_cast<const float4*>(c);
        y[0] = v.x; y[1] = v.y; y[2] = v.z; y[3] = v.w;
      } else {
#pragma unroll
        for (uint32_t k = 0; k < kLen; k++) { y[k] = c[k]; }
      }
      float d2 = 0.0f;
#pragma unroll
      for (uint32_t k = 0; k < kLen; k++) {
        const float d = __fsub_rn(r[s * kLen + k], y[k]);
        d2            = k == 0 ? __fmul_rn(d, d) : __fmaf_rn(d, d, d2);  // the chain starts from +0
      }
      if (d2 < best[s]) {
        best[s] = d2;
        code[s] = e;
      }
    };
#pragma unroll
    for (uint32_t s = 0; s < kSub; s++) {
      uint32_t pos = 0, stride = 1;
      bool in = s < nj;
#pragma unroll
      for (uint32_t k = 0; k < kLen; k++) {
        const float4 f = s_frame[s * kLen + k];
        const float2 e = s_ends[s * kLen + k];
        const float v = r[s * kLen + k], z = (v - f.x) * f.y, u = z * rsqrtf(1.0f + z * z);
        in          = in && v >= e.x && v <= e.y;
        const int p = min(max(int((u - f.z) * f.w), 0), int(kAxis) - 1);
        pos += uint32_t(p) * stride;
        stride *= kAxis;
      }
      from[s]        = (s * kCells + pos) * shape::bytes;
      const auto* cw = reinterpret_cast<const uint32_t*>(s_tables + (s < nj ? from[s] : 0u));
#pragma unroll
      for (uint32_t i = 0; i < kWords; i += 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(cw + i);
        cell[s][i] = v.x; cell[s][i + 1] = v.y;
      }
      if (!in) { cell[s][0] = kCellAll; }
      best[s] = INFINITY;
      code[s] = 0;
    }
#pragma unroll
    for (uint32_t q = 0; q < shape::sure; q++) {
#pragma unroll
      for (uint32_t s = 0; s < kSub; s++) {
        if ((cell[s][0] & 0xFFu) <= shape::codes) { look(s, (cell[s][(q + 1) / 4] >> (((q + 1) & 3u) * 8u)) & 0xFFu); }
      }
    }
#pragma unroll
    for (uint32_t s = 0; s < kSub; s++) {
      const uint32_t count = cell[s][0] & 0xFFu;
      if (count <= shape::codes) {
        for (uint32_t q = shape::sure; q < count; q++) { look(s, s_tables[from[s] + 1u + q]); }
      } else if (count == kCellLong) {
        const uint8_t* more = tables[j0 + s].spill + cell[s][1];
        for (uint32_t q = 0; q < ((cell[s][0] >> 8) & 0xFFu); q++) { look(s, __ldg(more + q)); }
      } else if (s < nj) {
        for (uint32_t e = 0; e < book; e++) { look(s, e); }
      }
    }
    uint8_t* o = codes + size_t(i) * pq_dim + j0;
    if (kSub == 4 && nj == 4 && (reinterpret_cast<uintptr_t>(o) & 3u) == 0) {
      uint32_t w = 0;
#pragma unroll
      for (uint32_t s = 0; s < kSub; s++) { w |= code[s] << (8u * s); }
      *reinterpret_cast<uint32_t*>(o) = w;
    } else {
#pragma unroll
      for (uint32_t s = 0; s < kSub; s++) {
        if (s < nj) { o[s] = uint8_t(code[s]); }
      }
    }
  }
}

// fn(std::integral_constant<uint32_t, components per subspace>) for the lengths that have tables of cells
template <typename Fn>
auto with_cell_len(uint32_t len, Fn&& fn)
{
  using std::integral_constant;
  switch (len) {
    case 1: return fn(integral_constant<uint32_t, 1>{});
    case 2: return fn(integral_constant<uint32_t, 2>{});
    case 3: return fn(integral_constant<uint32_t, 3>{});
    default: return fn(integral_constant<uint32_t, 4>{});
  }
}

// Byte codes of vectors taken in `order` -> interleaved list slots (and ids).  A warp handles 32 vectors and one 16-byte
// piece at a time: neighbours in a list are neighbours in the warp, so its stores are runs of 16-byte pieces.
__global__ void place_interleaved_kernel(const uint8_t* __restrict__ codes, const uint32_t* __restrict__ labels,
                                         const uint32_t* __restrict__ order, const uint32_t* __restrict__ slots, uint32_t n,
                                         uint32_t pq_dim, uint32_t bits, uint32_t n_pieces, const uint64_t* __restrict__ row_off,
                                         uint8_t* __restrict__ list_codes, int64_t* __restrict__ ids_out,
                                         const int64_t* __restrict__ src_ids, int64_t id_base)
{
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  const uint32_t i = blockIdx.x * 32u + lane;
  if (i >= n) { return; }
  const uint32_t row  = order ? order[i] : i;
  const uint64_t arow = row_off[labels[row]] + slots[i];
  const uint8_t* src  = codes + size_t(i) * pq_dim;
  const uint32_t cpp  = 128u / bits;
  for (uint32_t p = warp; p < n_pieces; p += n_warps) {
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (bits == 8u && p * 16u + 16u <= pq_dim && pq_dim % 16u == 0u) {
      const uint4 v = *reinterpret_cast<const uint4*>(src + p * 16u);
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else {
      const uint32_t nc = min(cpp, pq_dim - p * cpp);
      for (uint32_t t = 0; t < nc; t++) {
        const uint32_t code = src[p * cpp + t], bit = t * bits;
        w[bit >> 5] |= code << (bit & 31u);
        if ((bit & 31u) + bits > 32u) { w[(bit >> 5) + 1u] |= code >> (32u - (bit & 31u)); }
      }
    }
    *reinterpret_cast<uint4*>(list_codes + (((arow >> 5) * n_pieces + p) * 32u + (arow & 31u)) * 16u) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  if (warp == 0) { ids_out[arow] = src_ids ? src_ids[row] : id_base + int64_t(row); }
}

// Byte codes -> rows of a bit stream: plain output rows, or slots of FLAT lists (row_off given).  One thread per byte.
__global__ void place_flat_kernel(const uint8_t* __restrict__ codes, const uint32_t* __restrict__ labels,
                                  const uint32_t* __restrict__ order, const uint32_t* __restrict__ slots, uint32_t n,
                                  uint32_t pq_dim, uint32_t bits, uint32_t row_bytes, const uint64_t* __restrict__ row_off,
                                  uint8_t* __restrict__ out, int64_t* __restrict__ ids_out,
                                  const int64_t* __restrict__ src_ids, int64_t id_base)
{
  const uint64_t t = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (t >= uint64_t(n) * row_bytes) { return; }
  const uint32_t i = uint32_t(t / row_bytes), byte = uint32_t(t - uint64_t(i) * row_bytes);
  const uint32_t row = order ? order[i] : i;
  const uint8_t* src = codes + size_t(i) * pq_dim;
  uint32_t v         = 0;
  for (uint32_t j = (byte * 8u) / bits; j < pq_dim && j * bits < byte * 8u + 8u; j++) {
    const int shift     = int(j * bits) - int(byte * 8u);
    const uint32_t code = src[j];
    v |= shift >= 0 ? (code << shift) : (code >> (-shift));
  }
  uint64_t at = row;
  if (row_off) {
    at = row_off[labels[row]] + slots[i];
    if (byte == 0) { ids_out[at] = src_ids ? src_ids[row] : id_base + int64_t(row); }
  }
  out[at * row_bytes + byte] = uint8_t(v & 0xFFu);
}

// Codebooks per cluster: one warp per vector (taken in `order`): residual into shared memory, per-subspace argmin over the
// codebook split across lanes, then the lanes pack the codes.
//   interleaved != 0: write into the list arena at row (row_off[label] + slot[i]); ids too.
//   interleaved == 0: write a flat little-endian bit stream of ceil(pq_dim*bits/8) bytes per vector.
__global__ void encode_kernel(const float* __restrict__ x_ext, const uint32_t* __restrict__ labels,
                              const uint32_t* __restrict__ order, const uint32_t* __restrict__ slots,
                              uint32_t n, const float* __restrict__ centers,
                              const float* __restrict__ rot, int identity,
                              const float* __restrict__ pq_centers, uint32_t dim,
                              uint32_t dim_ext, uint32_t rot_dim, uint32_t pq_dim, uint32_t len,
                              uint32_t bits, int interleaved, const uint64_t* __restrict__ row_off,
                              uint8_t* __restrict__ codes_out, int64_t* __restrict__ ids_out,
                              const int64_t* __restrict__ src_ids, int64_t id_base,
                              uint32_t flat_row_bytes)
{
  extern __shared__ float s_enc[];
  const uint32_t warps = blockDim.x >> 5;
  const uint32_t wid   = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t per_warp_floats = round_up<uint32_t>(dim, 4) + round_up<uint32_t>(rot_dim, 4) + round_up<uint32_t>(pq_dim, 16) / 4;
  float* s_diff   = s_enc + size_t(wid) * per_warp_floats;
  float* s_res    = s_diff + round_up<uint32_t>(dim, 4);
  uint8_t* s_code = reinterpret_cast<uint8_t*>(s_res + round_up<uint32_t>(rot_dim, 4));
  const uint32_t i = blockIdx.x * warps + wid;
  if (i >= n) { return; }
  const uint32_t row   = order ? order[i] : i;
  const uint32_t label = labels[row];
  const uint32_t book  = 1u << bits;
  const float* x       = x_ext + size_t(row) * dim_ext;
  const float* c       = centers + size_t(label) * dim_ext;
  for (uint32_t k = lane; k < dim; k += 32) { s_diff[k] = __fsub_rn(x[k], c[k]); }
  __syncwarp();
  for (uint32_t r = lane; r < rot_dim; r += 32) {
    float acc;
    if (identity) {
      acc = s_diff[r];
    } else {
      const float* R = rot + size_t(r) * dim;
      acc            = 0.0f;
      for (uint32_t k = 0; k < dim; k++) { acc = __fmaf_rn(R[k], s_diff[k], acc); }
    }
    s_res[r] = acc;
  }
  __syncwarp();
  const float* pqc = pq_centers + size_t(label) * len * book;
  for (uint32_t j = 0; j < pq_dim; j++) {
    float best       = INFINITY;
    uint32_t best_b  = 0xFFFFFFFFu;
    for (uint32_t b = lane; b < book; b += 32) {
      float d2 = 0.0f;
      for (uint32_t k = 0; k < len; k++) {
        const float t = __fsub_rn(s_res[j * len + k], __ldg(pqc + size_t(k) * book + b));
        d2            = __fmaf_rn(t, t, d2);
      }
      if (d2 < best) {
        best   = d2;
        best_b = b;
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const float ob    = __shfl_xor_sync(kFullMask, best, d);
      const uint32_t oc = __shfl_xor_sync(kFullMask, best_b, d);
      if (ob < best || (ob == best && oc < best_b)) {
        best   = ob;
        best_b = oc;
      }
    }
    if (lane == 0) { s_code[j] = uint8_t(best_b == 0xFFFFFFFFu ? 0 : best_b); }
  }
  __syncwarp();
  if (interleaved == 1) {
    const uint32_t cpp      = 128u / bits;
    const uint32_t n_pieces = ceildiv(pq_dim, cpp);
    const uint64_t arow     = row_off[label] + slots[i];
    for (uint32_t p = lane; p < n_pieces; p += 32) {
      uint32_t w[4] = {0, 0, 0, 0};
      for (uint32_t t = 0; t < cpp && p * cpp + t < pq_dim; t++) {
        const uint32_t code = s_code[p * cpp + t];
        const uint32_t bit  = t * bits;
        w[bit >> 5] |= code << (bit & 31);
        if ((bit & 31) + bits > 32) { w[(bit >> 5) + 1] |= code >> (32 - (bit & 31)); }
      }
      uint4* dst = reinterpret_cast<uint4*>(codes_out + (((arow >> 5) * n_pieces + p) * 32 + (arow & 31)) * 16);
      *dst       = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (lane == 0) { ids_out[arow] = src_ids ? src_ids[row] : id_base + int64_t(row); }
  } else {
    // interleaved == 0: row `row` of a plain output matrix (transform); == 2: a slot of a FLAT list
    uint8_t* dst = codes_out + size_t(row) * flat_row_bytes;
    if (interleaved == 2) {
      const uint64_t arow = row_off[label] + slots[i];
      dst                 = codes_out + arow * flat_row_bytes;
      if (lane == 0) { ids_out[arow] = src_ids ? src_ids[row] : id_base + int64_t(row); }
    }
    for (uint32_t byte = lane; byte < flat_row_bytes; byte += 32) {
      uint32_t v = 0;
      // collect the bits [byte*8, byte*8+8) of the stream
      const uint32_t first = (byte * 8) / bits;
      for (uint32_t j = first; j < pq_dim && j * bits < byte * 8 + 8; j++) {
        const int shift = int(j * bits) - int(byte * 8);
        const uint32_t code = s_code[j];
        v |= shift >= 0 ? (code << shift) : (code >> (-shift));
      }
      dst[byte] = uint8_t(v & 0xFFu);
    }
  }
}

// Interleaved list rows [offset, offset + n) -> flat bit-packed rows.
__global__ void unpack_contiguous_kernel(const uint8_t* __restrict__ list, uint32_t n, uint32_t offset,
                                         uint32_t pq_dim, uint32_t bits, uint32_t flat_row_bytes,
                                         uint8_t* __restrict__ out)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) { return; }
  const uint32_t row      = offset + i;
  const uint32_t cpp      = 128u / bits;
  const uint32_t n_pieces = ceildiv(pq_dim, cpp);
  uint8_t* dst            = out + size_t(i) * flat_row_bytes;
  for (uint32_t b = 0; b < flat_row_bytes; b++) { dst[b] = 0; }
  for (uint32_t j = 0; j < pq_dim; j++) {
    const uint32_t p = j / cpp, t = j % cpp;
    const uint8_t* piece = list + ((size_t(row >> 5) * n_pieces + p) * 32 + (row & 31)) * 16;
    const uint32_t bit   = t * bits;
    uint32_t pair        = piece[bit >> 3];
    if ((bit & 7) + bits > 8) { pair |= uint32_t(piece[(bit >> 3) + 1]) << 8; }
    const uint32_t code = (pair >> (bit & 7)) & ((1u << bits) - 1u);
    const uint32_t ob   = j * bits;
    dst[ob >> 3] |= uint8_t((code << (ob & 7)) & 0xFFu);
    if ((ob & 7) + bits > 8) { dst[(ob >> 3) + 1] |= uint8_t(code >> (8 - (ob & 7))); }
  }
}

// Code j of one interleaved list row.
__device__ __forceinline__ uint32_t list_code(const uint8_t* __restrict__ list, uint32_t row, uint32_t j,
                                              uint32_t n_pieces, uint32_t bits)
{
  const uint32_t cpp = 128u / bits;
  const uint32_t p = j / cpp, bit = (j % cpp) * bits;
  const uint8_t* piece = list + ((size_t(row >> 5) * n_pieces + p) * 32 + (row & 31)) * 16;
  uint32_t pair        = piece[bit >> 3];
  if ((bit & 7) + bits > 8) { pair |= uint32_t(piece[(bit >> 3) + 1]) << 8; }
  return (pair >> (bit & 7)) & ((1u << bits) - 1u);
}

// One thread per (row, subspace): interleaved list rows -> one code per byte.
__global__ void unpack_codes_kernel(const uint8_t* __restrict__ list, uint32_t n, uint32_t offset,
                                    const uint32_t* __restrict__ indices, uint32_t pq_dim, uint32_t bits,
                                    uint32_t n_pieces, uint8_t* __restrict__ out)
{
  const uint64_t t = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (t >= uint64_t(n) * pq_dim) { return; }
  const uint32_t i = uint32_t(t / pq_dim), j = uint32_t(t % pq_dim);
  const uint32_t row = indices ? indices[i] : offset + i;
  out[t] = uint8_t(list_code(list, row, j, n_pieces, bits));
}

// One thread per (row, 16-byte piece): codes (one per byte, or bit-packed rows when kContiguous)
// -> interleaved list rows [offset, offset + n).  Unused bits of the last piece are zero.
template <bool kContiguous>
__global__ void pack_codes_kernel(const uint8_t* __restrict__ codes, uint32_t n, uint32_t offset,
                                  uint32_t pq_dim, uint32_t bits, uint32_t n_pieces,
                                  uint32_t flat_row_bytes, uint8_t* __restrict__ list)
{
  const uint64_t t = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (t >= uint64_t(n) * n_pieces) { return; }
  const uint32_t i = uint32_t(t / n_pieces), p = uint32_t(t % n_pieces);
  const uint32_t cpp = 128u / bits, mask = (1u << bits) - 1u;
  const uint8_t* src = codes + size_t(i) * (kContiguous ? flat_row_bytes : pq_dim);
  uint32_t w[4] = {0, 0, 0, 0};
  for (uint32_t c = 0; c < cpp && p * cpp + c < pq_dim; c++) {
    const uint32_t j = p * cpp + c;
    uint32_t code;
    if (kContiguous) {
      const uint32_t ib = j * bits;
      uint32_t pair     = src[ib >> 3];
      if ((ib & 7) + bits > 8) { pair |= uint32_t(src[(ib >> 3) + 1]) << 8; }
      code = (pair >> (ib & 7)) & mask;
    } else {
      code = src[j] & mask;
    }
    const uint32_t bit = c * bits;
    w[bit >> 5] |= code << (bit & 31);
    if ((bit & 31) + bits > 32) { w[(bit >> 5) + 1] |= code >> (32 - (bit & 31)); }
  }
  const uint32_t row = offset + i;
  *reinterpret_cast<uint4*>(list + ((size_t(row >> 5) * n_pieces + p) * 32 + (row & 31)) * 16) =
    make_uint4(w[0], w[1], w[2], w[3]);
}

template <typename T>
__device__ __forceinline__ T from_float(float x);
template <> __device__ __forceinline__ float from_float<float>(float x) { return x; }
template <> __device__ __forceinline__ __half from_float<__half>(float x) { return __float2half_rn(x); }
// mapping<int8_t>(float) clamps before it converts (ann_utils.cuh:211-217); the uint8 mapping does not
template <> __device__ __forceinline__ int8_t from_float<int8_t>(float x)
{
  return static_cast<int8_t>(fminf(fmaxf(__fmul_rn(x, 128.0f), -128.0f), 127.0f));
}
template <> __device__ __forceinline__ uint8_t from_float<uint8_t>(float x) { return static_cast<uint8_t>(__fmul_rn(x, 256.0f)); }

// One block per row: decode the row in the rotated space (codeword + rotated list center, one add
// per component), then out[i, d] = sum over r, in order, of rotation[r, d] * decoded[r] (fp32 fma).
template <typename T>
__global__ void reconstruct_kernel(const uint8_t* __restrict__ list, uint32_t offset,
                                   const uint32_t* __restrict__ indices, const float* __restrict__ pq_centers,
                                   int per_cluster, const float* __restrict__ center_rot,
                                   const float* __restrict__ rot, uint32_t label, uint32_t dim,
                                   uint32_t rot_dim, uint32_t pq_dim, uint32_t len, uint32_t bits,
                                   uint32_t n_pieces, T* __restrict__ out)
{
  extern __shared__ float s_dec[];
  const uint32_t i    = blockIdx.x;
  const uint32_t row  = indices ? indices[i] : offset + i;
  const uint32_t book = 1u << bits;
  for (uint32_t r = threadIdx.x; r < rot_dim; r += blockDim.x) {
    const uint32_t j = r / len, k = r % len;
    const uint32_t code = list_code(list, row, j, n_pieces, bits);
    const float* pqc    = pq_centers + size_t(per_cluster ? label : j) * len * book;
    s_dec[r]            = __fadd_rn(pqc[size_t(k) * book + code], center_rot[r]);
  }
  __syncthreads();
  for (uint32_t d = threadIdx.x; d < dim; d += blockDim.x) {
    float acc = 0.0f;
    for (uint32_t r = 0; r < rot_dim; r++) { acc = __fmaf_rn(rot[size_t(r) * dim + d], s_dec[r], acc); }
    out[size_t(i) * dim + d] = from_float<T>(acc);
  }
}

__global__ void fill_u32_kernel(uint32_t* p, uint32_t n, uint32_t v)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { p[i] = v; }
}

__global__ void add_scalar_u32_kernel(uint32_t* p, uint32_t n, uint32_t v)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { p[i] += v; }
}

// ------------------------------------------------------------------------------------------------
// extend helpers
// ------------------------------------------------------------------------------------------------
__global__ void histogram_kernel(const uint32_t* __restrict__ labels, uint64_t n, uint32_t* __restrict__ counts)
{
  const uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (i < n) { atomicAdd(counts + labels[i], 1u); }
}

__global__ void iota_kernel(uint32_t* p, uint32_t n)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { p[i] = i; }
}

// slots[i] = base[label] + (i - first index of label in the sorted order)
__global__ void slots_kernel(const uint32_t* __restrict__ sorted_labels, uint32_t n,
                             const uint32_t* __restrict__ base, uint32_t* __restrict__ slots)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) { return; }
  const uint32_t l = sorted_labels[i];
  // first position of l: binary search for the lower bound
  uint32_t lo = 0, hi = i;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (sorted_labels[mid] < l) {
      lo = mid + 1;
    } else {
      hi = mid;
    }
  }
  slots[i] = base[l] + (i - lo);
}

// One block per list: copy the old list payload (whole 32-row groups) and ids to the new arena.
__global__ void relocate_lists_kernel(const uint8_t* __restrict__ old_codes, const int64_t* __restrict__ old_ids,
                                      const uint64_t* __restrict__ old_off, const uint32_t* __restrict__ old_sizes,
                                      const uint64_t* __restrict__ new_off, uint32_t row_bytes,
                                      uint8_t* __restrict__ new_codes, int64_t* __restrict__ new_ids)
{
  const uint32_t l = blockIdx.x;
  const uint32_t n = old_sizes[l];
  if (n == 0) { return; }
  const uint64_t rows  = round_up<uint64_t>(n, 32);
  const uint4* src     = reinterpret_cast<const uint4*>(old_codes + old_off[l] * row_bytes);
  uint4* dst           = reinterpret_cast<uint4*>(new_codes + new_off[l] * row_bytes);
  const uint64_t n_vec = rows * row_bytes / 16;
  for (uint64_t i = threadIdx.x; i < n_vec; i += blockDim.x) { dst[i] = src[i]; }
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) { new_ids[new_off[l] + i] = old_ids[old_off[l] + i]; }
}

uint64_t chunk_rows_for(uint32_t dim_ext)
{
  const uint64_t budget = 1ull << 29;  // bytes of converted rows per chunk
  return std::max<uint64_t>(1024, std::min<uint64_t>(1u << 19, budget / (uint64_t(dim_ext) * 4)));
}

// balanced k-means defaults of the reference (cpp/include/cuvs/cluster/kmeans.hpp:181-204)
constexpr double kBalanceLower  = 0.333;
constexpr double kBalanceUpper  = 3.0;
constexpr float kCentroidOffset = 0.01f;

struct label_ctx {
  float alpha;
  float pad;
  bool normalize;
};
label_ctx labeling_of(DistanceType m)
{
  // IP trains/predicts with L2 (ivf_pq_build.cuh:70-76); cosine works on normalised rows.
  return {-2.0f, -0.5f, m == DistanceType::CosineExpanded};
}

// Labelling of many rows against one set of centres: on the tensor cores (label_tc.cu) where there is enough work to fill
// them, else by the exact product.  Works in memory that the caller provides, on any number of rows.
class nearest_labeler {
 public:
  static size_t bytes(const raft::resources& res, uint64_t n_rows, uint32_t n_lists, uint32_t dim)
  {
    const uint32_t batch = batch_of(n_rows);
    return label_tc_usable(batch, n_lists)
             ? round_up<size_t>(label_model_bytes(n_lists, dim, true), 256) + label_workspace_bytes(res, batch, n_lists, dim)
             : size_t(batch) * 8;
  }
  // `dim`: index of the |c|^2 column of the centre rows (rows carry -0.5 there); n_rows: the most that run() is given
  nearest_labeler(raft::resources& res, const float* centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                  float alpha, uint64_t n_rows, void* mem)
    : res_(res), centers_(centers), n_lists_(n_lists), dim_(dim), dim_ext_(dim_ext), batch_(batch_of(n_rows)), alpha_(alpha),
      use_tc_(label_tc_usable(batch_, n_lists)), mem_(static_cast<char*>(mem))
  {
    refresh();
  }
  // the centres have changed
  void refresh()
  {
    if (!use_tc_) { return; }
    prepare_label_model(res_.stream, centers_, n_lists_, dim_, dim_ext_, 0.5f, true, mem_);
    res_.launches += 3;
  }
  // labels[i] = nearest list of row i of x_ext [n_rows, dim_ext]
  void run(const float* x_ext, uint64_t n_rows, uint32_t* labels)
  {
    for (uint64_t r0 = 0; r0 < n_rows; r0 += batch_) {
      const uint32_t nr = uint32_t(std::min<uint64_t>(batch_, n_rows - r0));
      const float* x    = x_ext + r0 * dim_ext_;
      if (use_tc_) {
        label_rows_tc(res_, centers_, mem_, n_lists_, dim_, dim_ext_, alpha_, x, nr, labels + r0,
                      mem_ + round_up<size_t>(label_model_bytes(n_lists_, dim_, true), 256));
      } else {
        assign_nearest(res_, centers_, n_lists_, dim_ext_, alpha_, x, nr, labels + r0, reinterpret_cast<unsigned long long*>(mem_));
      }
    }
  }

 private:
  static uint32_t batch_of(uint64_t n_rows) { return uint32_t(std::min<uint64_t>(n_rows, 1u << 19)); }
  raft::resources& res_;
  const float* centers_;
  uint32_t n_lists_, dim_, dim_ext_, batch_;
  float alpha_;
  bool use_tc_;
  char* mem_;
};

// Host rows -> device staging (no-op for device data).
const void* stage_rows(raft::resources& res, const void* data, elem_t t, uint64_t r0, uint64_t nr,
                       uint32_t dim, bool on_device, void* staging)
{
  const size_t es = elem_size(t);
  const char* src = static_cast<const char*>(data) + r0 * dim * es;
  if (on_device) { return src; }
  CUDA_TRY(cudaMemcpyAsync(staging, src, nr * dim * es, cudaMemcpyHostToDevice, res.stream));
  return staging;
}

void make_rotation(uint32_t rot_dim, uint32_t dim, bool force_random, std::vector<float>& out)
{
  out.assign(size_t(rot_dim) * dim, 0.0f);
  if (rot_dim == dim && !force_random) {
    for (uint32_t i = 0; i < dim; i++) { out[size_t(i) * dim + i] = 1.0f; }
    return;
  }
  // random orthogonal: Gaussian matrix, columns orthonormalised (modified Gram-Schmidt, twice)
  const uint32_t n = rot_dim;
  std::vector<double> a(size_t(n) * n);
  std::mt19937_64 gen(7);
  std::normal_distribution<double> nd(0.0, 1.0);
  for (auto& v : a) { v = nd(gen); }
  for (uint32_t c = 0; c < n; c++) {
    for (int pass = 0; pass < 2; pass++) {
      for (uint32_t p = 0; p < c; p++) {
        double dot = 0;
        for (uint32_t r = 0; r < n; r++) { dot += a[size_t(r) * n + c] * a[size_t(r) * n + p]; }
        for (uint32_t r = 0; r < n; r++) { a[size_t(r) * n + c] -= dot * a[size_t(r) * n + p]; }
      }
    }
    double nn = 0;
    for (uint32_t r = 0; r < n; r++) { nn += a[size_t(r) * n + c] * a[size_t(r) * n + c]; }
    nn = std::sqrt(nn);
    for (uint32_t r = 0; r < n; r++) { a[size_t(r) * n + c] /= nn; }
  }
  for (uint32_t r = 0; r < rot_dim; r++) {
    for (uint32_t c = 0; c < dim; c++) { out[size_t(r) * dim + c] = float(a[size_t(r) * n + c]); }
  }
}

// Whether n vectors are encoded through tables of cells: where making those costs less than they save.  What a vector saves grows with
// the subspaces, and so does the making of the tables beyond what a handful of them takes; few codewords (7 bits) leave less to save:
// the two sides meet at some a + b / pq_dim vectors.  Whole calls of `transform` by comparing all / through tables (us), 256 codewords:
// 64 subspaces of one component 112 / 107 at 24,576 vectors, 163 / 125 at 49,152; of two 166 / 154 and 261 / 196; of three 437 / 481 at
// 65,536, 786 / 614 at 131,072; of four 998 / 1,310 at 131,072, 1,929 / 1,541 at 262,144; 16 subspaces of two 95 / 96 and, unit vectors,
// 93 / 114 at 24,576, 128 / 113 at 40,000; 8 of four 331 / 467 at 262,144, 610 / 560 at 524,288; 2 of two 85 / 90 at 98,304.  128
// codewords, 64 subspaces of two: 135 / 146 at 24,576, 202 / 182 at 49,152.
bool encode_by_cells(const index<int64_t>& idx, uint64_t n)
{
  const uint32_t len = idx.pq_len(), bits = idx.pq_bits();
  if (idx.codebook_kind() != codebook_gen::PER_SUBSPACE || len > 4 || bits < 7) { return false; }
  constexpr uint32_t kFixed[2][4] = {{25'000, 22'000, 100'000, 170'000}, {12'000, 14'000, 60'000, 175'000}};
  constexpr uint32_t kShared[2][4] = {{1'000'000, 800'000, 1'500'000, 2'300'000}, {200'000, 250'000, 1'300'000, 2'600'000}};
  // (four to eight subspaces leave the comparison of all too few blocks)
  if (bits == 8 && len <= 2 && idx.pq_dim() >= 4 && idx.pq_dim() <= 8) { return n >= 24'576; }
  return n >= kFixed[bits - 7][len - 1] + kShared[bits - 7][len - 1] / idx.pq_dim();
}
size_t code_table_bytes(const index<int64_t>& idx)
{
  return idx.pq_dim() * with_cell_len(idx.pq_len(), [](auto len) { return sizeof(code_table<decltype(len)::value>); });
}
// Scratch of launch_encode for up to n vectors: the tables of cells, at an offset that does not depend on n (the chunks of a call
// after the first find them there, so nothing may write them in between), byte codes, and with a rotation the differences before
// and after it.
size_t encode_scratch_bytes(const index<int64_t>& idx, uint64_t n, bool cells)
{
  if (idx.codebook_kind() == codebook_gen::PER_CLUSTER) { return 0; }
  ws_layout lay;
  if (cells) { lay.add(code_table_bytes(idx)); }
  lay.add(n * idx.pq_dim());
  if (!idx.rotation_is_identity()) {
    lay.add(n * idx.dim() * 4);
    lay.add(n * idx.rot_dim() * 4);
  }
  return lay.total();
}

// `to_lists`: write slots of the index's lists (and ids); else plain rows of codes_out.  `cells`: through tables of cells, made
// first where make_tables is set (else they are in `scratch` from the call before).
void launch_encode(raft::resources& res, const index<int64_t>& idx, const float* x_ext,
                   const uint32_t* labels, const uint32_t* order, const uint32_t* slots, uint32_t n,
                   bool to_lists, uint8_t* codes_out, int64_t* ids_out, const int64_t* src_ids,
                   int64_t id_base, void* scratch, bool cells, bool make_tables)
{
  if (n == 0) { return; }
  const uint32_t row_bytes = ceildiv(idx.pq_dim() * idx.pq_bits(), 8u);
  const bool flat          = !to_lists || idx.codes_layout() == list_layout::FLAT;
  if (idx.codebook_kind() == codebook_gen::PER_CLUSTER) {
    const uint32_t warps = 4;
    const uint32_t per_warp_floats = round_up<uint32_t>(idx.dim(), 4) + round_up<uint32_t>(idx.rot_dim(), 4) +
                                     round_up<uint32_t>(idx.pq_dim(), 16) / 4;
    const size_t smem = size_t(warps) * per_warp_floats * 4;
    CUVS_EXPECTS(smem <= 48 * 1024, "dim = %u is too large for the encoder", idx.dim());
    encode_kernel<<<ceildiv(n, warps), warps * 32, smem, res.stream>>>(
      x_ext, labels, order, slots, n, idx.centers(), idx.rotation_matrix(), idx.rotation_is_identity(),
      idx.pq_centers(), idx.dim(), idx.dim_ext(), idx.rot_dim(), idx.pq_dim(), idx.pq_len(), idx.pq_bits(),
      // 0: rows of a plain output matrix; 1: slots of interleaved lists; 2: slots of flat lists
      to_lists ? (flat ? 2 : 1) : 0, idx.row_offsets(), codes_out, ids_out, src_ids, id_base, row_bytes);
    CUDA_TRY(cudaGetLastError());
    res.launches++;
    return;
  }
  const uint32_t dim = idx.dim(), dim_ext = idx.dim_ext(), rot_dim = idx.rot_dim(), len = idx.pq_len();
  const uint32_t pq_dim = idx.pq_dim(), book = idx.pq_book_size();
  ws_layout lay;
  char* ws     = static_cast<char*>(scratch);
  void* tables = cells ? ws + lay.add(code_table_bytes(idx)) : nullptr;
  auto* bytes  = reinterpret_cast<uint8_t*>(ws + lay.add(size_t(n) * pq_dim));
  // plain rows of 8-bit codes are the byte codes themselves
  const bool direct = !to_lists && idx.pq_bits() == 8;
  if (direct) { bytes = codes_out; }
  const float* x        = x_ext;
  uint32_t x_stride     = dim_ext;
  const float* c        = idx.centers();
  const uint32_t* x_order = order;
  if (!idx.rotation_is_identity()) {
    auto* diff  = reinterpret_cast<float*>(ws + lay.add(size_t(n) * dim * 4));
    auto* resid = reinterpret_cast<float*>(ws + lay.add(size_t(n) * rot_dim * 4));
    difference_kernel<<<unsigned(ceildiv<uint64_t>(uint64_t(n) * dim, 256)), 256, 0, res.stream>>>(
      x_ext, labels, order, idx.centers(), n, dim, dim_ext, diff);
    exact_rows_product(res, idx.rotation_matrix(), rot_dim, diff, n, dim, dim, 1.0f, resid);
    res.launches++;
    x        = resid;
    x_stride = rot_dim;
    c        = nullptr;
    x_order  = nullptr;
  }
  auto go = [&](auto lenc) {
    constexpr uint32_t kLen = decltype(lenc)::value;
    constexpr uint32_t kSub = enc_subspaces<kLen>();
    const size_t need  = size_t(kSub) * len * book * 4;
    const bool in_smem = need <= 96 * 1024;
    if (in_smem) { ensure_dynamic_smem(reinterpret_cast<const void*>(encode_subspaces_kernel<kLen>), need); }
    const dim3 grid(ceildiv(n, 256u * kEncVecs), ceildiv(pq_dim, kSub));
    encode_subspaces_kernel<kLen><<<grid, 256, in_smem ? need : 0, res.stream>>>(
      x, x_stride, x_order, labels, c, dim_ext, n, idx.pq_centers(), pq_dim, len, book, in_smem, bytes, pq_dim);
    CUDA_TRY(cudaGetLastError());
  };
  auto go_cells = [&](auto lenc) {
    constexpr uint32_t kLen = decltype(lenc)::value;
    using shape             = cell_shape<kLen>;
    auto* tab               = static_cast<code_table<kLen>*>(tables);
    if (make_tables) {
      CUDA_TRY(cudaMemset2DAsync(&tab->n_spill, sizeof(*tab), 0, 4, pq_dim, res.stream));
      code_cells_kernel<kLen><<<dim3(pq_dim, kCells / 256), 256, 0, res.stream>>>(idx.pq_centers(), book, tab);
      res.launches++;
    }
    const size_t smem = size_t(shape::subs) * (kCells * shape::bytes + book * kLen * 4);
    ensure_dynamic_smem(reinterpret_cast<const void*>(encode_cells_kernel<kLen>), smem);
    // about two blocks per SM, each reading its tables once
    const uint32_t groups = ceildiv(pq_dim, shape::subs);
    const uint32_t shares = std::max(1u, 2u * uint32_t(res.sm_count) / groups);
    const uint32_t rows   = round_up(ceildiv(n, shares), 1024u);
    const bool vec        = x_stride % 4 == 0 && dim_ext % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    encode_cells_kernel<kLen><<<dim3(groups, ceildiv(n, rows)), 1024, smem, res.stream>>>(
      x, x_stride, x_order, labels, c, dim_ext, n, idx.pq_centers(), tab, pq_dim, book, rows, vec, bytes);
    CUDA_TRY(cudaGetLastError());
  };
  using std::integral_constant;
  if (cells) {
    with_cell_len(len, go_cells);
  } else {
    switch (len) {
      case 1: go(integral_constant<uint32_t, 1>{}); break;
      case 2: go(integral_constant<uint32_t, 2>{}); break;
      case 3: go(integral_constant<uint32_t, 3>{}); break;
      case 4: go(integral_constant<uint32_t, 4>{}); break;
      case 8: go(integral_constant<uint32_t, 8>{}); break;
      default: go(integral_constant<uint32_t, 0>{});
    }
  }
  res.launches++;
  if (direct) { return; }
  if (flat) {
    place_flat_kernel<<<unsigned(ceildiv<uint64_t>(uint64_t(n) * row_bytes, 256)), 256, 0, res.stream>>>(
      bytes, labels, order, slots, n, pq_dim, idx.pq_bits(), row_bytes, to_lists ? idx.row_offsets() : nullptr, codes_out,
      ids_out, src_ids, id_base);
  } else {
    const uint32_t warps = std::min<uint32_t>(8, idx.n_pieces());
    place_interleaved_kernel<<<ceildiv(n, 32u), warps * 32, 0, res.stream>>>(bytes, labels, order, slots, n, pq_dim, idx.pq_bits(),
                                                                            idx.n_pieces(), idx.row_offsets(), codes_out,
                                                                            ids_out, src_ids, id_base);
  }
  CUDA_TRY(cudaGetLastError());
  res.launches++;
}

// Re-create the arenas for `new_sizes`, keeping the first min(old, new) rows (codes and ids) of every list.
void resize_lists(raft::resources& res, index<int64_t>* idx, const std::vector<uint32_t>& new_sizes)
{
  const uint32_t n_lists    = idx->n_lists();
  const cudaStream_t stream = res.stream;
  std::vector<uint32_t> keep(n_lists);
  bool any = false;
  for (uint32_t l = 0; l < n_lists; l++) {
    keep[l] = std::min(idx->host_list_sizes()[l], new_sizes[l]);
    any |= keep[l] > 0;
  }
  if (!any) {
    idx->allocate_lists(new_sizes, stream);
    return;
  }
  dev_array<uint8_t> old_codes = std::move(idx->codes_);
  dev_array<int64_t> old_ids   = std::move(idx->ids_);
  dev_array<uint64_t> old_off(size_t(n_lists) + 1);
  dev_array<uint32_t> keep_d(n_lists);
  CUDA_TRY(cudaMemcpyAsync(old_off.data(), idx->row_offsets(), (size_t(n_lists) + 1) * 8, cudaMemcpyDeviceToDevice, stream));
  CUDA_TRY(cudaMemcpyAsync(keep_d.data(), keep.data(), size_t(n_lists) * 4, cudaMemcpyHostToDevice, stream));
  idx->allocate_lists(new_sizes, stream);
  relocate_lists_kernel<<<n_lists, 128, 0, stream>>>(old_codes.data(), old_ids.data(), old_off.data(),
                                                     keep_d.data(), idx->row_offsets(),
                                                     idx->list_row_bytes(), idx->codes(), idx->ids());
  CUDA_TRY(cudaGetLastError());
  res.launches++;
  res.sync();  // the old arenas are released on return
}

}  // namespace

// ------------------------------------------------------------------------------------------------
// helpers
// ------------------------------------------------------------------------------------------------
namespace helpers {

void unpack_contiguous_list_data(raft::resources& res, const index<int64_t>& idx, uint8_t* out_codes,
                                 uint32_t n_rows, uint32_t label, uint32_t offset)
{
  CUVS_EXPECTS(label < idx.n_lists(), "label %u is out of range", label);
  CUVS_EXPECTS(uint64_t(offset) + n_rows <= idx.host_list_sizes()[label],
               "rows [%u, %u) exceed the size of list %u (%u)", offset, offset + n_rows, label,
               idx.host_list_sizes()[label]);
  if (n_rows == 0) { return; }
  if (idx.codes_layout() == list_layout::FLAT) {
    // the rows already are what the caller asks for
    const size_t bpv = idx.bytes_per_vector();
    CUDA_TRY(cudaMemcpyAsync(out_codes, idx.codes() + (idx.host_row_offsets()[label] + offset) * bpv,
                             size_t(n_rows) * bpv, cudaMemcpyDeviceToDevice, res.stream));
    return;
  }
  const uint8_t* list = idx.codes() + idx.host_row_offsets()[label] * size_t(idx.n_pieces()) * 16;
  unpack_contiguous_kernel<<<ceildiv(n_rows, 128u), 128, 0, res.stream>>>(
    list, n_rows, offset, idx.pq_dim(), idx.pq_bits(), ceildiv(idx.pq_dim() * idx.pq_bits(), 8u), out_codes);
  CUDA_TRY(cudaGetLastError());
  res.launches++;
}

void set_model(raft::resources& res, index<int64_t>* idx, const float* pq_centers, const float* centers,
               uint32_t centers_cols, const float* centers_rot, const float* rotation_matrix)
{
  CUDA_TRY(cudaMemcpyAsync(idx->pq_centers(), pq_centers, idx->pq_centers_size() * 4,
                           cudaMemcpyDefault, res.stream));
  if (centers_cols == idx->dim_ext()) {
    CUDA_TRY(cudaMemcpyAsync(idx->centers(), centers, size_t(idx->n_lists()) * idx->dim_ext() * 4,
                             cudaMemcpyDefault, res.stream));
  } else {
    pad_centers_kernel<<<ceildiv(idx->n_lists(), 128u), 128, 0, res.stream>>>(
      centers, idx->n_lists(), idx->dim(), idx->dim_ext(), idx->centers());
    res.launches++;
  }
  CUDA_TRY(cudaMemcpyAsync(idx->centers_rot(), centers_rot, size_t(idx->n_lists()) * idx->rot_dim() * 4,
                           cudaMemcpyDefault, res.stream));
  CUDA_TRY(cudaMemcpyAsync(idx->rotation_matrix(), rotation_matrix,
                           size_t(idx->rot_dim()) * idx->dim() * 4, cudaMemcpyDefault, res.stream));
  res.sync();
  idx->allocate_lists(std::vector<uint32_t>(idx->n_lists(), 0), res.stream);
  idx->recompute_model_state(res.stream);
}

namespace {
void check_rows(const index<int64_t>& idx, uint32_t label, uint32_t offset, uint32_t n_rows)
{
  CUVS_EXPECTS(label < idx.n_lists(), "label %u is out of range", label);
  // ivf_pq_build.cuh:611-612
  CUVS_EXPECTS(uint64_t(offset) + n_rows <= idx.host_list_sizes()[label],
               "offset + output size must be not bigger than the cluster size.");
}
uint8_t* list_base(const index<int64_t>& idx, uint32_t label)
{
  // the helpers that read or write single codes address the interleaved layout (as the reference's do)
  CUVS_EXPECTS(idx.codes_layout() == list_layout::INTERLEAVED,
               "this helper supports the INTERLEAVED codes layout only");
  return idx.codes() + idx.host_row_offsets()[label] * size_t(idx.n_pieces()) * kIndexGroupVecLen;
}
// Grow list `label` by n_rows, write the new source ids; returns the first new row.
uint32_t extend_list_prepare(raft::resources& res, index<int64_t>* idx, const int64_t* new_indices,
                             uint32_t n_rows, uint32_t label)
{
  CUVS_EXPECTS(idx != nullptr && label < idx->n_lists(), "label %u is out of range", label);
  const uint32_t offset = idx->host_list_sizes()[label];
  CUVS_EXPECTS(uint64_t(offset) + n_rows < (1ull << 32), "list %u grows beyond 2^32 rows", label);
  std::vector<uint32_t> sizes = idx->host_list_sizes();
  sizes[label] += n_rows;
  resize_lists(res, idx, sizes);
  CUDA_TRY(cudaMemcpyAsync(idx->ids() + idx->host_row_offsets()[label] + offset, new_indices,
                           size_t(n_rows) * 8, cudaMemcpyDefault, res.stream));
  return offset;
}
}  // namespace

namespace codepacker {

void unpack_list_data(raft::resources& res, const index<int64_t>& idx, uint8_t* out_codes,
                      uint32_t n_rows, uint32_t label, uint32_t offset,
                      const uint32_t* in_cluster_indices)
{
  check_rows(idx, label, in_cluster_indices ? 0 : offset, in_cluster_indices ? 0 : n_rows);
  if (n_rows == 0) { return; }
  const uint64_t n_threads = uint64_t(n_rows) * idx.pq_dim();
  unpack_codes_kernel<<<unsigned(ceildiv<uint64_t>(n_threads, 256)), 256, 0, res.stream>>>(
    list_base(idx, label), n_rows, offset, in_cluster_indices, idx.pq_dim(), idx.pq_bits(),
    idx.n_pieces(), out_codes);
  CUDA_TRY(cudaGetLastError());
  res.launches++;
}

namespace {
template <bool kContiguous>
void pack_rows(raft::resources& res, index<int64_t>* idx, const uint8_t* codes, uint32_t n_rows,
               uint32_t label, uint32_t offset)
{
  CUVS_EXPECTS(idx != nullptr, "null index");
  check_rows(*idx, label, offset, n_rows);
  if (n_rows == 0) { return; }
  if (kContiguous && idx->codes_layout() == list_layout::FLAT) {
    const size_t bpv = idx->bytes_per_vector();
    CUDA_TRY(cudaMemcpyAsync(idx->codes() + (idx->host_row_offsets()[label] + offset) * bpv, codes,
                             size_t(n_rows) * bpv, cudaMemcpyDefault, res.stream));
    return;
  }
  const uint64_t n_threads = uint64_t(n_rows) * idx->n_pieces();
  pack_codes_kernel<kContiguous><<<unsigned(ceildiv<uint64_t>(n_threads, 256)), 256, 0, res.stream>>>(
    codes, n_rows, offset, idx->pq_dim(), idx->pq_bits(), idx->n_pieces(),
    ceildiv(idx->pq_dim() * idx->pq_bits(), 8u), list_base(*idx, label));
  CUDA_TRY(cudaGetLastError());
  res.launches++;
}
}  // namespace

void pack_list_data(raft::resources& res, index<int64_t>* idx, const uint8_t* codes, uint32_t n_rows,
                    uint32_t label, uint32_t offset)
{
  pack_rows<false>(res, idx, codes, n_rows, label, offset);
}

void pack_contiguous_list_data(raft::resources& res, index<int64_t>* idx, const uint8_t* codes,
                               uint32_t n_rows, uint32_t label, uint32_t offset)
{
  pack_rows<true>(res, idx, codes, n_rows, label, offset);
}

void reconstruct_list_data(raft::resources& res, const index<int64_t>& idx, void* out_vectors,
                           elem_t out_type, uint32_t n_rows, uint32_t label, uint32_t offset,
                           const uint32_t* in_cluster_indices)
{
  if (n_rows == 0) { return; }
  check_rows(idx, label, in_cluster_indices ? 0 : offset, in_cluster_indices ? 0 : n_rows);
  const size_t smem = size_t(idx.rot_dim()) * 4;
  CUVS_EXPECTS(smem <= 48 * 1024, "rot_dim = %u is too large to reconstruct", idx.rot_dim());
  auto launch = [&](auto* out) {
    using T = std::remove_pointer_t<decltype(out)>;
    reconstruct_kernel<T><<<n_rows, 128, smem, res.stream>>>(
      list_base(idx, label), offset, in_cluster_indices, idx.pq_centers(),
      idx.codebook_kind() == codebook_gen::PER_CLUSTER, idx.centers_rot() + size_t(label) * idx.rot_dim(),
      idx.rotation_matrix(), label, idx.dim(), idx.rot_dim(), idx.pq_dim(), idx.pq_len(), idx.pq_bits(),
      idx.n_pieces(), out);
  };
  switch (out_type) {
    case elem_t::f32: launch(static_cast<float*>(out_vectors)); break;
    case elem_t::f16: launch(static_cast<__half*>(out_vectors)); break;
    case elem_t::i8: launch(static_cast<int8_t*>(out_vectors)); break;
    default: launch(static_cast<uint8_t*>(out_vectors));
  }
  CUDA_TRY(cudaGetLastError());
  res.launches++;
}

void extend_list_with_codes(raft::resources& res, index<int64_t>* idx, const uint8_t* new_codes,
                            const int64_t* new_indices, uint32_t n_rows, uint32_t label)
{
  const uint32_t offset = extend_list_prepare(res, idx, new_indices, n_rows, label);
  pack_rows<false>(res, idx, new_codes, n_rows, label, offset);
  res.sync();
}

void extend_list_with_contiguous_codes(raft::resources& res, index<int64_t>* idx,
                                       const uint8_t* new_codes, const int64_t* new_indices,
                                       uint32_t n_rows, uint32_t label)
{
  const uint32_t offset = extend_list_prepare(res, idx, new_indices, n_rows, label);
  pack_rows<true>(res, idx, new_codes, n_rows, label, offset);
  res.sync();
}

void extend_list(raft::resources& res, index<int64_t>* idx, const void* new_vectors, elem_t dtype,
                 const int64_t* new_indices, uint32_t n_rows, uint32_t label)
{
  const uint32_t offset = extend_list_prepare(res, idx, new_indices, n_rows, label);
  if (n_rows == 0) { return; }
  const label_ctx lc = labeling_of(idx->metric());
  dev_array<float> x_ext(size_t(n_rows) * idx->dim_ext());
  dev_array<uint32_t> labels(n_rows), slots(n_rows);
  dev_array<uint8_t> scratch(encode_scratch_bytes(*idx, n_rows, false));
  to_float_ext(res, new_vectors, dtype, n_rows, 1, idx->dim(), idx->dim_ext(), lc.pad, lc.normalize,
               x_ext.data());
  fill_u32_kernel<<<ceildiv(n_rows, 256u), 256, 0, res.stream>>>(labels.data(), n_rows, label);
  iota_kernel<<<ceildiv(n_rows, 256u), 256, 0, res.stream>>>(slots.data(), n_rows);
  add_scalar_u32_kernel<<<ceildiv(n_rows, 256u), 256, 0, res.stream>>>(slots.data(), n_rows, offset);
  res.launches += 3;
  // ids were written by extend_list_prepare: the encoder gets the same array, so it rewrites them
  launch_encode(res, *idx, x_ext.data(), labels.data(), nullptr, slots.data(), n_rows, true, idx->codes(),
                idx->ids(), new_indices, 0, scratch.data(), false, false);
  res.sync();
}

}  // namespace codepacker

void erase_list(raft::resources& res, index<int64_t>* idx, uint32_t label)
{
  CUVS_EXPECTS(idx != nullptr && label < idx->n_lists(), "label %u is out of range", label);
  std::vector<uint32_t> sizes = idx->host_list_sizes();
  sizes[label]                = 0;
  resize_lists(res, idx, sizes);
}

void reset_index(raft::resources& res, index<int64_t>* idx)
{
  CUVS_EXPECTS(idx != nullptr, "null index");
  idx->allocate_lists(std::vector<uint32_t>(idx->n_lists(), 0), res.stream);
}

}  // namespace helpers

// ------------------------------------------------------------------------------------------------
// extend
// ------------------------------------------------------------------------------------------------
void extend_any(raft::resources& res, const void* new_vectors, elem_t dtype, int64_t n_rows_i,
                const int64_t* new_indices, bool on_device, index<int64_t>* idx)
{
  CUVS_EXPECTS(idx != nullptr && idx->n_lists() > 0, "extend: the index is not trained");
  CUVS_EXPECTS(n_rows_i >= 0 && n_rows_i < (1ll << 32), "extend: unsupported number of rows");
  // ivf_pq_build.cuh:1011-1012
  CUVS_EXPECTS(new_indices != nullptr || idx->size() == 0,
               "You must pass data indices when the index is non-empty.");
  const uint64_t n = uint64_t(n_rows_i);
  if (n == 0) { return; }
  const cudaStream_t stream = res.stream;
  const uint32_t dim = idx->dim(), dim_ext = idx->dim_ext(), n_lists = idx->n_lists();
  const label_ctx lc   = labeling_of(idx->metric());
  const uint64_t chunk = std::min<uint64_t>(n, chunk_rows_for(dim_ext));
  const bool cells     = encode_by_cells(*idx, n);

  int end_bit = 1;
  while ((1ull << end_bit) < n_lists) { end_bit++; }
  size_t cub_bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                  static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr), int(chunk), 0, end_bit, stream);
  // one grow-only scratch buffer of the handle for everything below (a dozen allocations and releases per call took as
  // long as the work on 300,000 rows)
  ws_layout lay;
  const size_t row_bytes = size_t(dim) * elem_size(dtype);
  const size_t o_x       = lay.add(chunk * dim_ext * 4);
  // (the labels of more rows than these are released on return: they grow with the call, not with its chunks)
  constexpr uint64_t kKeptLabels = 1ull << 26;
  dev_array<uint32_t> many_labels(n > kKeptLabels ? n : 0);
  const size_t o_labels  = lay.add(n > kKeptLabels ? 0 : n * 4);
  const size_t o_counts  = lay.add(size_t(n_lists) * 4);
  const size_t o_fill    = lay.add(size_t(n_lists) * 4);
  const size_t o_iota    = lay.add(chunk * 4);
  const size_t o_order   = lay.add(chunk * 4);
  const size_t o_sorted  = lay.add(chunk * 4);
  const size_t o_slots   = lay.add(chunk * 4);
  const size_t o_cub     = lay.add(cub_bytes);
  const size_t o_staging = lay.add(on_device ? 0 : chunk * row_bytes);
  const size_t o_ids     = lay.add(on_device || !new_indices ? 0 : chunk * 8);
  // (labelling and encoding take turns)
  const size_t o_work    = lay.add(std::max(nearest_labeler::bytes(res, chunk, n_lists, dim), encode_scratch_bytes(*idx, chunk, cells)));
  res.scratch.reserve(lay.total());
  char* ws        = res.scratch.base();
  auto* x_ext     = reinterpret_cast<float*>(ws + o_x);
  auto* labels    = n > kKeptLabels ? many_labels.data() : reinterpret_cast<uint32_t*>(ws + o_labels);
  auto* counts    = reinterpret_cast<uint32_t*>(ws + o_counts);
  auto* fill      = reinterpret_cast<uint32_t*>(ws + o_fill);  // rows already placed in each list
  auto* iota      = reinterpret_cast<uint32_t*>(ws + o_iota);
  auto* order     = reinterpret_cast<uint32_t*>(ws + o_order);
  auto* sorted    = reinterpret_cast<uint32_t*>(ws + o_sorted);
  auto* slots     = reinterpret_cast<uint32_t*>(ws + o_slots);
  void* staging   = ws + o_staging;
  CUDA_TRY(cudaMemsetAsync(counts, 0, size_t(n_lists) * 4, stream));

  // pass 1: labels + histogram
  {
    nearest_labeler labeler(res, idx->centers(), n_lists, dim, dim_ext, lc.alpha, chunk, ws + o_work);
    for (uint64_t r0 = 0; r0 < n; r0 += chunk) {
      const uint64_t nr = std::min(chunk, n - r0);
      const void* src   = stage_rows(res, new_vectors, dtype, r0, nr, dim, on_device, staging);
      to_float_ext(res, src, dtype, nr, 1, dim, dim_ext, lc.pad, lc.normalize, x_ext);
      labeler.run(x_ext, nr, labels + r0);
    }
  }
  histogram_kernel<<<unsigned(ceildiv<uint64_t>(n, 256)), 256, 0, stream>>>(labels, n, counts);
  std::vector<uint32_t> h_counts(n_lists);
  CUDA_TRY(cudaMemcpyAsync(h_counts.data(), counts, size_t(n_lists) * 4, cudaMemcpyDeviceToHost, stream));
  res.sync();

  // new arenas, old payload moved over
  std::vector<uint32_t> old_sizes = idx->host_list_sizes();
  std::vector<uint32_t> new_sizes(n_lists);
  for (uint32_t l = 0; l < n_lists; l++) {
    CUVS_EXPECTS(uint64_t(old_sizes[l]) + h_counts[l] < (1ull << 32), "list %u grows beyond 2^32 rows", l);
    new_sizes[l] = old_sizes[l] + h_counts[l];
  }
  resize_lists(res, idx, new_sizes);

  // pass 2: per chunk, order rows by list (stable), give each its slot, encode
  CUDA_TRY(cudaMemcpyAsync(fill, old_sizes.data(), size_t(n_lists) * 4, cudaMemcpyHostToDevice, stream));
  for (uint64_t r0 = 0; r0 < n; r0 += chunk) {
    const uint32_t nr = uint32_t(std::min(chunk, n - r0));
    if (n > chunk) {  // (else the rows of pass 1 are still there)
      const void* src = stage_rows(res, new_vectors, dtype, r0, nr, dim, on_device, staging);
      to_float_ext(res, src, dtype, nr, 1, dim, dim_ext, lc.pad, lc.normalize, x_ext);
    }
    iota_kernel<<<ceildiv(nr, 256u), 256, 0, stream>>>(iota, nr);
    cub::DeviceRadixSort::SortPairs(ws + o_cub, cub_bytes, labels + r0, sorted, iota, order, int(nr), 0, end_bit, stream);
    slots_kernel<<<ceildiv(nr, 256u), 256, 0, stream>>>(sorted, nr, fill, slots);
    const int64_t* ids_chunk = new_indices ? new_indices + r0 : nullptr;
    if (new_indices && !on_device) {
      CUDA_TRY(cudaMemcpyAsync(ws + o_ids, new_indices + r0, size_t(nr) * 8, cudaMemcpyHostToDevice, stream));
      ids_chunk = reinterpret_cast<const int64_t*>(ws + o_ids);
    }
    launch_encode(res, *idx, x_ext, labels + r0, order, slots, nr, true, idx->codes(), idx->ids(), ids_chunk, int64_t(r0),
                  ws + o_work, cells, r0 == 0);
    if (r0 + chunk < n) {
      // rows of the chunk are placed
      histogram_kernel<<<ceildiv(nr, 256u), 256, 0, stream>>>(labels + r0, nr, fill);
      res.launches++;
    }
    CUDA_TRY(cudaGetLastError());
    res.launches += 3;
  }
  res.sync();
}

// ------------------------------------------------------------------------------------------------
// transform
// ------------------------------------------------------------------------------------------------
void transform_any(raft::resources& res, const index<int64_t>& idx, const void* dataset, elem_t dtype,
                   int64_t n_rows_i, uint32_t* out_labels, uint8_t* out_codes)
{
  CUVS_EXPECTS(n_rows_i >= 0 && n_rows_i < (1ll << 32), "transform: unsupported number of rows");
  const uint64_t n = uint64_t(n_rows_i);
  if (n == 0) { return; }
  const uint32_t dim = idx.dim(), dim_ext = idx.dim_ext();
  const label_ctx lc   = labeling_of(idx.metric());
  const uint64_t chunk = std::min<uint64_t>(n, chunk_rows_for(dim_ext));
  const bool cells     = encode_by_cells(idx, n);
  const uint32_t flat  = ceildiv(idx.pq_dim() * idx.pq_bits(), 8u);
  ws_layout lay;
  const size_t o_x     = lay.add(chunk * dim_ext * 4);
  const size_t o_label = lay.add(nearest_labeler::bytes(res, chunk, idx.n_lists(), dim));
  const size_t o_enc   = lay.add(encode_scratch_bytes(idx, chunk, cells));
  res.scratch.reserve(lay.total());
  char* ws    = res.scratch.base();
  auto* x_ext = reinterpret_cast<float*>(ws + o_x);
  nearest_labeler labeler(res, idx.centers(), idx.n_lists(), dim, dim_ext, lc.alpha, chunk, ws + o_label);
  for (uint64_t r0 = 0; r0 < n; r0 += chunk) {
    const uint32_t nr = uint32_t(std::min(chunk, n - r0));
    const char* src   = static_cast<const char*>(dataset) + r0 * dim * elem_size(dtype);
    to_float_ext(res, src, dtype, nr, 1, dim, dim_ext, lc.pad, lc.normalize, x_ext);
    labeler.run(x_ext, nr, out_labels + r0);
    launch_encode(res, idx, x_ext, out_labels + r0, nullptr, nullptr, nr, false, out_codes + r0 * flat, nullptr, nullptr, 0,
                  ws + o_enc, cells, r0 == 0);
  }
  res.sync();
}

// ------------------------------------------------------------------------------------------------
// build
// ------------------------------------------------------------------------------------------------
void build_any(raft::resources& res, const index_params& params, const void* dataset, elem_t dtype,
               int64_t n_rows_i, uint32_t dim, bool on_device, index<int64_t>* out)
{
  CUVS_EXPECTS(n_rows_i > 0 && dim > 0, "build: empty dataset");
  CUVS_EXPECTS(params.n_lists > 0, "n_lists must be positive");
  const uint64_t n_rows     = uint64_t(n_rows_i);
  const cudaStream_t stream = res.stream;
  index<int64_t> idx(params.metric, params.codebook_kind, params.n_lists, dim, params.pq_bits,
                     params.pq_dim, params.conservative_memory_allocation, params.codes_layout);
  const uint32_t n_lists = idx.n_lists(), dim_ext = idx.dim_ext(), rot_dim = idx.rot_dim();
  const uint32_t book = idx.pq_book_size(), len = idx.pq_len(), pq_dim = idx.pq_dim();
  const label_ctx lc  = labeling_of(idx.metric());

  // ---- trainset (ivf_pq_build.cuh:1283-1290): every `stride`-th row ----
  const double frac      = std::min(1.0, std::max(0.0, params.kmeans_trainset_fraction));
  const uint64_t want    = std::max<uint64_t>(uint64_t(frac * double(n_rows)), n_lists);
  const uint64_t stride  = std::max<uint64_t>(1, n_rows / std::max<uint64_t>(1, want));
  const uint64_t n_train = n_rows / stride;
  CUVS_EXPECTS(n_train < (1ull << 32), "trainset too large");
  dev_array<float> train(n_train * dim_ext);
  {
    dev_array<uint8_t> staging;
    const void* src = dataset;
    if (!on_device) {
      const size_t rb = size_t(dim) * elem_size(dtype);
      staging.resize(n_train * rb);
      CUDA_TRY(cudaMemcpy2DAsync(staging.data(), rb, dataset, rb * stride, rb, n_train,
                                 cudaMemcpyHostToDevice, stream));
      src = staging.data();
      to_float_ext(res, src, dtype, n_train, 1, dim, dim_ext, lc.pad, lc.normalize, train.data());
      res.sync();
    } else {
      to_float_ext(res, src, dtype, n_train, stride, dim, dim_ext, lc.pad, lc.normalize, train.data());
    }
  }

  // ---- coarse k-means ----
  dev_array<uint32_t> labels(n_train);
  dev_array<uint8_t> label_mem(nearest_labeler::bytes(res, n_train, n_lists, dim));
  dev_array<float> sums(size_t(n_lists) * dim);
  dev_array<uint32_t> counts(n_lists);
  init_centers_kernel<<<n_lists, 128, 0, stream>>>(train.data(), n_train, n_lists, dim_ext, idx.centers());
  center_norms_kernel<<<ceildiv(n_lists, 128u), 128, 0, stream>>>(idx.centers(), n_lists, dim, dim_ext);
  res.launches += 2;
  const uint32_t iters = std::max<uint32_t>(1, params.kmeans_n_iters);
  nearest_labeler labeler(res, idx.centers(), n_lists, dim, dim_ext, lc.alpha, n_train, label_mem.data());
  for (uint32_t it = 0; it < iters; it++) {
    labeler.refresh();
    labeler.run(train.data(), n_train, labels.data());
    CUDA_TRY(cudaMemsetAsync(sums.data(), 0, sums.size() * 4, stream));
    CUDA_TRY(cudaMemsetAsync(counts.data(), 0, size_t(n_lists) * 4, stream));
    accumulate_kernel<<<unsigned(ceildiv<uint64_t>(n_train * 32, 256)), 256, 0, stream>>>(
      train.data(), labels.data(), n_train, dim, dim_ext, sums.data(), counts.data());
    finalize_centers_kernel<<<n_lists, 128, 0, stream>>>(sums.data(), counts.data(), dim, dim_ext,
                                                         train.data(), n_train, it + 1, lc.normalize,
                                                         idx.centers());
    CUDA_TRY(cudaGetLastError());
    res.launches += 2;
    // Balancing (not after the last step, whose means are final): clusters sorted by size, the i-th
    // smallest paired with the i-th largest; where the small one is underfull (< 1/3 of the average)
    // or the large one overfull (> 3 x the average), the small one restarts next to the large one.
    if (it + 1 < iters && n_lists >= 2) {
      std::vector<uint32_t> h_counts(n_lists);
      CUDA_TRY(cudaMemcpyAsync(h_counts.data(), counts.data(), size_t(n_lists) * 4, cudaMemcpyDeviceToHost, stream));
      res.sync();
      std::vector<uint32_t> order(n_lists);
      for (uint32_t l = 0; l < n_lists; l++) { order[l] = l; }
      std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
        return h_counts[a] != h_counts[b] ? h_counts[a] < h_counts[b] : a < b;
      });
      const double avg = double(n_train) / double(n_lists);
      std::vector<uint32_t> h_pairs;
      for (uint32_t i = 0; i < n_lists / 2; i++) {
        const uint32_t small = order[i], large = order[n_lists - 1 - i];
        const bool underfull = double(h_counts[small]) < avg * kBalanceLower;
        const bool overfull  = double(h_counts[large]) > avg * kBalanceUpper;
        if (!underfull && !overfull) { break; }  // sizes are sorted: no later pair qualifies either
        if (h_counts[large] < 2) { break; }
        h_pairs.push_back(small);
        h_pairs.push_back(large);
      }
      if (!h_pairs.empty()) {
        dev_array<uint32_t> d_pairs(h_pairs.size());
        dev_array<unsigned long long> member(n_lists);
        CUDA_TRY(cudaMemcpyAsync(d_pairs.data(), h_pairs.data(), h_pairs.size() * 4, cudaMemcpyHostToDevice, stream));
        CUDA_TRY(cudaMemsetAsync(member.data(), 0, size_t(n_lists) * 8, stream));
        pick_member_kernel<<<unsigned(ceildiv<uint64_t>(n_train, 256)), 256, 0, stream>>>(labels.data(), n_train,
                                                                                         it + 1, member.data());
        adjust_centers_kernel<<<unsigned(h_pairs.size() / 2), 128, 0, stream>>>(
          idx.centers(), d_pairs.data(), member.data(), train.data(), dim, dim_ext, kCentroidOffset, lc.normalize);
        CUDA_TRY(cudaGetLastError());
        res.sync();  // the pair list and the member table are released here
        res.launches += 2;
      }
    }
  }
  labeler.refresh();
  labeler.run(train.data(), n_train, labels.data());

  // ---- rotation, rotated centers ----
  {
    std::vector<float> rot;
    make_rotation(rot_dim, dim, params.force_random_rotation, rot);
    CUDA_TRY(cudaMemcpyAsync(idx.rotation_matrix(), rot.data(), rot.size() * 4, cudaMemcpyHostToDevice, stream));
    res.sync();
  }
  rotate_centers_kernel<<<unsigned(ceildiv<uint64_t>(uint64_t(n_lists) * rot_dim, 256)), 256, 0, stream>>>(
    idx.centers(), idx.rotation_matrix(), n_lists, dim, dim_ext, rot_dim, idx.centers_rot());
  res.launches++;
  idx.allocate_lists(std::vector<uint32_t>(n_lists, 0), stream);
  idx.detect_identity_rotation(stream);

  // ---- PQ codebooks ----
  {
    const uint64_t max_pts = uint64_t(std::max<uint32_t>(1, params.max_train_points_per_pq_code)) * book;
    const bool per_cluster = idx.codebook_kind() == codebook_gen::PER_CLUSTER;
    const uint64_t n_pq    = per_cluster ? n_train : std::min<uint64_t>(n_train, max_pts);
    const uint64_t pstride = std::max<uint64_t>(1, n_train / n_pq);
    dev_array<float> resid(n_pq * rot_dim);
    residual_kernel<<<unsigned(n_pq), 128, size_t(dim) * 4, stream>>>(
      train.data(), labels.data(), pstride, idx.centers(), idx.rotation_matrix(),
      idx.rotation_is_identity(), dim, dim_ext, rot_dim, resid.data());
    res.launches++;
    const size_t smem = size_t(book) * len * 8 + size_t(book) * 4;
    CUVS_EXPECTS(smem <= 200 * 1024, "pq_len = %u is too large for codebook training", len);
    ensure_dynamic_smem(reinterpret_cast<const void*>(train_codebooks_kernel), smem);
    const int pq_iters = 25;
    if (!per_cluster) {
      train_codebooks_kernel<<<pq_dim, 1024, smem, stream>>>(resid.data(), uint32_t(n_pq), rot_dim, pq_dim,
                                                             len, book, 0, nullptr, nullptr, 0, pq_iters,
                                                             idx.pq_centers());
    } else {
      // rows of each list: stable sort of the trainset labels
      dev_array<uint32_t> iota(n_train), order(n_train), sorted_labels(n_train), begin(size_t(n_lists) + 1);
      iota_kernel<<<unsigned(ceildiv<uint64_t>(n_train, 256)), 256, 0, stream>>>(iota.data(), uint32_t(n_train));
      size_t cub_bytes = 0;
      int end_bit      = 1;
      while ((1ull << end_bit) < n_lists) { end_bit++; }
      cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, labels.data(), sorted_labels.data(), iota.data(),
                                      order.data(), int(n_train), 0, end_bit, stream);
      dev_array<uint8_t> tmp(cub_bytes);
      cub::DeviceRadixSort::SortPairs(tmp.data(), cub_bytes, labels.data(), sorted_labels.data(), iota.data(),
                                      order.data(), int(n_train), 0, end_bit, stream);
      CUDA_TRY(cudaMemsetAsync(begin.data(), 0, (size_t(n_lists) + 1) * 4, stream));
      histogram_kernel<<<unsigned(ceildiv<uint64_t>(n_train, 256)), 256, 0, stream>>>(labels.data(), n_train, begin.data());
      std::vector<uint32_t> hb(size_t(n_lists) + 1);
      CUDA_TRY(cudaMemcpyAsync(hb.data(), begin.data(), (size_t(n_lists) + 1) * 4, cudaMemcpyDeviceToHost, stream));
      res.sync();
      uint32_t run = 0;
      for (uint32_t l = 0; l <= n_lists; l++) {
        uint32_t c = hb[l];
        hb[l]      = run;
        run += (l < n_lists ? c : 0);
      }
      CUDA_TRY(cudaMemcpyAsync(begin.data(), hb.data(), (size_t(n_lists) + 1) * 4, cudaMemcpyHostToDevice, stream));
      const uint32_t max_rows = uint32_t(std::max<uint64_t>(1, ceildiv<uint64_t>(max_pts, pq_dim)));
      train_codebooks_kernel<<<n_lists, 256, smem, stream>>>(resid.data(), uint32_t(n_pq), rot_dim, pq_dim,
                                                             len, book, 1, order.data(), begin.data(),
                                                             max_rows, pq_iters, idx.pq_centers());
      res.sync();
    }
    CUDA_TRY(cudaGetLastError());
    res.launches++;
    res.sync();
  }

  idx.recompute_model_state(stream);

  // ---- fill ----
  if (params.add_data_on_build) {
    train.reset();
    extend_any(res, dataset, dtype, n_rows_i, nullptr, on_device, &idx);
  }
  *out = std::move(idx);
}

}  // namespace cuvs::neighbors::ivf_pq
