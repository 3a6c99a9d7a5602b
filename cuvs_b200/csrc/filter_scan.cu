// The bounding pass of the fine search: approximate scores of every (query, row of a probed list) on the
// tensor cores, reduced to one value per eight rows.
//
// Reference: compute_similarity scores every row of every probed list through a per-pair look-up table
// (cpp/src/neighbors/ivf_pq/ivf_pq_search.cuh:526-644).  A table costs pq_dim * 2^bits entries per pair and a
// gather per code and row; nearly all of the rows so scored cannot reach the k best.  Here a list is decoded
// once for up to 128 queries that probe it: its rows become a half-precision operand in shared memory
// (K-major, 128-byte swizzle), the queries' differences to the list centre the other one, and
//     L2:  |r|^2 - 2 (q - c).r        inner product:  -q.r
// comes out of tcgen05.mma for 128 x 256 (query, row) pairs at a time; |r|^2 rides in three extra columns
// (two halfs of it, and a mask for rows that do not count).  Epilogue warps (thread = query) keep the
// minimum of every eight rows, add the pair's constant and store it.  rescore.cu turns these values into
// rigorous bounds and scores exactly what they leave.
//
// A tile is eight 32-row groups -- of one list, or of several short ones whose pairs are neighbours -- so that
// lists of a few rows and queries fill it.
// The query operand of every (query, list) pair is written once, ordered by list, by pair_operands_kernel and
// comes in by TMA.  Warp roles of the persistent CTA (one per SM): warps 0-15 decode (two threads per row of the
// list, each half of every K block), 16-23 are the epilogue (lane quarter = warp % 4, two warps per quarter), 24 issues the MMAs,
// 25 the TMA loads.  K is cut into blocks of 64 halfs that pass through a ring of stages (query block 16 KB, row block
// 32 KB); two TMEM accumulators let the epilogue of a tile overlap the next one.  Every wait is bounded: on a
// time-out the kernel raises the error word and returns, and rescore.cu then scores every row.
//
// What bounds it: for few queries per list the gathers of the decode (one 4-byte look-up per code for two
// dimensions per subspace, 3.4 wavefronts each on random codes); for many, the epilogue and the operand feed.
#include "common.hpp"
#include "filter_scan.hpp"
#include "packed.cuh"
#include "search_internal.hpp"
#include "tc_ptx.cuh"
#include "topk.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace cuvs::neighbors::ivf_pq {

using namespace cuvs_b200;

namespace {

constexpr uint32_t kTileQ    = 128;
constexpr uint32_t kTileR    = 256;
constexpr uint32_t kBlockK   = 64;                      // halfs per K block: one 128-byte swizzle atom
constexpr uint32_t kABytes   = kTileQ * kBlockK * 2;    // 16 KB
constexpr uint32_t kBBytes   = kTileR * kBlockK * 2;    // 32 KB
constexpr uint32_t kStage    = kABytes + kBBytes;
constexpr uint32_t kMaxStages = 4;
constexpr uint32_t kDecodeWarps = 16, kEpiWarp = 16, kEpiWarps = 8, kMmaWarp = 24, kTmaWarp = 25;
constexpr uint32_t kFilterThreads = 26 * 32;
constexpr float kMaskHalf    = 32768.0f;                // mask x mask = 2^30 in the scaled domain

// acc += h * h in fp32 (the half widens exactly)
__device__ __forceinline__ float fma_half_sq(uint32_t h2, bool hi, float acc)
{
  if (hi) {
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tfma.rn.f32.f16 %0, h, h, %0;\n\t}" : "+f"(acc) : "r"(h2));
  } else {
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tfma.rn.f32.f16 %0, l, l, %0;\n\t}" : "+f"(acc) : "r"(h2));
  }
  return acc;
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y)
{
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ uint32_t half2_bits(float a, float b)
{
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// Look-ups in the codebook at [address + constant]: its contents do not change, so these may move freely.
template <uint32_t kOff>
__device__ __forceinline__ uint32_t lds32(uint32_t a)
{
  uint32_t v;
  asm("ld.shared.b32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(kOff));
  return v;
}
template <uint32_t kOff>
__device__ __forceinline__ uint32_t lds16(uint32_t a)
{
  uint16_t v;
  asm("ld.shared.b16 %0, [%1+%2];" : "=h"(v) : "r"(a), "n"(kOff));
  return v;
}
template <uint32_t kOff>
__device__ __forceinline__ void lds64(uint32_t a, uint32_t& x, uint32_t& y)
{
  asm("ld.shared.v2.b32 {%0, %1}, [%2+%3];" : "=r"(x), "=r"(y) : "r"(a), "n"(kOff));
}
template <uint32_t kOff>
__device__ __forceinline__ void lds128(uint32_t a, uint32_t& x, uint32_t& y, uint32_t& z, uint32_t& w)
{
  asm("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4+%5];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(a), "n"(kOff));
}
// byte offset of 16-byte chunk c (0..7) of row r inside a swizzled K block
__device__ __forceinline__ uint32_t swz(uint32_t r, uint32_t c) { return r * 128u + ((c ^ (r & 7u)) << 4); }


// kBits 8 or 4 (kWords): the codes of half a K block are extracted from whole words with constant shifts; other widths,
// and subspaces of more than eight components, code by code.  kLP: halfs per subspace in the K layout (1, 2, 4 or 8;
// without kWords 8 stands for every multiple of 8).
template <int kBits, int kLP, bool kWords, bool kCodes>
__global__ void __launch_bounds__(kFilterThreads, 1)
filter_kernel(const __grid_constant__ CUtensorMap map_16, const __grid_constant__ CUtensorMap map_64,
              const __grid_constant__ CUtensorMap map_128, const filter_params p)
{
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_a  = smem_u32(smem_raw);
  const uint32_t base_a = (raw_a + 1023u) & ~1023u;
  uint8_t* base_p       = smem_raw + (base_a - raw_a);
  const uint32_t book_a = base_a + p.n_stages * kStage;
  uint64_t* bars        = reinterpret_cast<uint64_t*>(base_p + p.n_stages * kStage + p.book_bytes);
  const uint32_t bar_full   = smem_u32(bars);
  const uint32_t bar_empty  = bar_full + kMaxStages * 8;
  const uint32_t bar_tfull  = bar_empty + kMaxStages * 8;
  const uint32_t bar_tempty = bar_tfull + 2 * 8;
  uint32_t* tmem_slot       = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 4);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t n_blocks = (p.k_chunks + 7u) >> 3;

  // (barriers, tensor memory and the codebook, which is the index's: while the kernel before this one ends)
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < p.n_stages; s++) {
      mbar_init(bar_full + s * 8, kDecodeWarps + 1);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (uint32_t a = 0; a < 2; a++) {
      mbar_init(bar_tfull + a * 8, 1);
      mbar_init(bar_tempty + a * 8, kEpiWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(p.book);
    uint4* dst       = reinterpret_cast<uint4*>(base_p + p.n_stages * kStage);
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < p.book_bytes / 16; i += kFilterThreads) { dst[i] = __ldg(src + i); }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_begin();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const uint32_t n_tiles   = __ldg(p.n_tiles);
  bool ok = true;

  if (warp < kDecodeWarps) {
    // ---------------- rows of the list -> operand B ----------------
    // warps 2i and 2i + 1 share the 32 rows of group i: chunks 0-3 and 4-7 of every K block
    constexpr uint32_t kCodes = kLP >= 8 ? 4u : 32u / kLP;            // codes per half block
    constexpr uint32_t kNW    = !kWords ? 1u : (kCodes * kBits + 31u) / 32u;      // their words
    constexpr uint32_t kCPC   = kLP >= 8 ? 1u : 8u / kLP;             // codes per chunk
    [[maybe_unused]] constexpr uint32_t kSubStep = (1u << kBits) * 2u * kLP;  // bytes of a subspace's codebook
    const uint32_t r        = (warp >> 1) * 32u + lane, half = warp & 1u;
    const uint32_t eb       = 2u * p.len_pad;                // bytes of a codebook entry
    const uint32_t sub_step = p.book_size * eb;              // bytes of a subspace's codebook
    // (the words of the next K block are on their way while one is decoded)
    uint32_t stage = 0, phase = 0;
    const uint32_t gi = warp >> 1;
    struct group_ref {
      uint32_t arena;   // first row / 32
      uint32_t n_rows;  // 0: no rows of this tile are this warp's
    };
    auto group_of = [&](uint32_t t) -> group_ref {
      group_ref g{0u, 0u};
      if (t < n_tiles && gi < __ldg(&p.tiles[t].n_groups)) {
        const uint2 d = __ldg(reinterpret_cast<const uint2*>(&p.tiles[t].group[gi]));
        g.arena       = d.x;
        g.n_rows      = d.y & 0xFFu;
      }
      return g;
    };
    const uint8_t* lane_src = p.codes + lane * 16u;
    auto src_of = [&](const group_ref& g) { return lane_src + uint64_t(g.arena) * (p.n_pieces * 512u); };
    // the words that hold this thread's codes of K block kb
    auto load_words = [&](const group_ref& g, uint32_t kb, uint32_t (&w)[kNW]) {
      if constexpr (kWords) {
        constexpr uint32_t kBytes = kCodes * kBits / 8u;       // per half block: 2 .. 32
        const uint32_t byte  = (kb * 2u + half) * kBytes;      // in the row's code stream
        const uint32_t piece = byte >> 4;
        if (g.n_rows != 0u && piece < p.n_pieces) {
          const uint8_t* a = src_of(g) + (piece * 512u + (byte & 15u));
          if constexpr (kBytes == 32) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(a));
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
            if (piece + 1 < p.n_pieces) {
              const uint4 u = __ldg(reinterpret_cast<const uint4*>(a + 512));
              w[4] = u.x; w[5] = u.y; w[6] = u.z; w[7] = u.w;
            }
          } else if constexpr (kBytes == 16) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(a));
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
          } else if constexpr (kBytes == 8) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(a));
            w[0] = v.x; w[1] = v.y;
          } else if constexpr (kBytes == 4) {
            w[0] = __ldg(reinterpret_cast<const uint32_t*>(a));
          } else {
            w[0] = __ldg(reinterpret_cast<const uint16_t*>(a));
          }
        }
      }
    };
    // the four chunks of this thread of K block kb
    auto look = [&](const group_ref& g, uint32_t kb, const uint32_t (&w)[kNW], uint32_t (&h)[4][4]) {
      if (g.n_rows == 0u) { return; }
      const uint32_t g0 = kb * 8u + half * 4u;
      if constexpr (!kWords) {
        // code j, from the piece that holds it
        uint32_t have      = 0xFFFFFFFFu;
        uint4 pv           = make_uint4(0u, 0u, 0u, 0u);
        constexpr uint32_t cpp = 128u / kBits;
        auto code_at       = [&](uint32_t j) -> uint32_t {
          const uint32_t piece = j / cpp, bit = (j - piece * cpp) * kBits;
          if (piece != have) {
            pv   = __ldg(reinterpret_cast<const uint4*>(src_of(g) + piece * 512u));
            have = piece;
          }
          const uint32_t lo = bit < 64u ? (bit < 32u ? pv.x : pv.y) : (bit < 96u ? pv.z : pv.w);
          const uint32_t hi = bit < 64u ? (bit < 32u ? pv.y : pv.z) : pv.w;
          return __funnelshift_r(lo, hi, bit & 31u) & ((1u << kBits) - 1u);
        };
#pragma unroll
        for (uint32_t c = 0; c < 4; c++) {
          h[c][0] = h[c][1] = h[c][2] = h[c][3] = 0u;
          if (g0 + c >= p.data_chunks) { continue; }
          if constexpr (kLP == 8) {
            // entries of len_pad / 8 chunks
            const uint32_t m = p.len_pad / 8u, j = (g0 + c) / m, sub = (g0 + c) - j * m;
            lds128<0>(book_a + j * sub_step + code_at(j) * eb + sub * 16u, h[c][0], h[c][1], h[c][2], h[c][3]);
          } else {
            const uint32_t j = (g0 + c) * kCPC;
#pragma unroll
            for (uint32_t i = 0; i < kCPC; i++) {
              if (j + i >= p.pq_dim) { continue; }
              const uint32_t at = book_a + (j + i) * sub_step + code_at(j + i) * (2u * kLP);
              if constexpr (kLP == 1) { h[c][i >> 1] |= lds16<0>(at) << ((i & 1u) * 16u); }
              if constexpr (kLP == 2) { h[c][i] = lds32<0>(at); }
              if constexpr (kLP == 4) { lds64<0>(at, h[c][2 * i], h[c][2 * i + 1]); }
            }
          }
        }
      } else {
        // entry of the n-th code of this thread's half block
        const uint32_t base_j = book_a + g0 * kCPC * kSubStep;
        auto code_of = [&](auto nc) -> uint32_t {
          constexpr uint32_t n = decltype(nc)::value;
          if constexpr (kBits == 8) {
            return __byte_perm(w[n >> 2], 0u, 0x4440u + (n & 3u));
          } else {
            return (w[n >> 3] >> ((n & 7u) * 4u)) & 15u;
          }
        };
        auto look_up = [&](auto nc) {
          constexpr uint32_t n = decltype(nc)::value, c = n / kCPC, i = n % kCPC;
          const uint32_t at    = base_j + code_of(nc) * (2u * kLP);
          if constexpr (kLP == 1) {
            const uint32_t v = lds16<n * kSubStep>(at);
            h[c][i >> 1]     = (i & 1u) ? (h[c][i >> 1] | (v << 16)) : v;
          }
          if constexpr (kLP == 2) { h[c][i] = lds32<n * kSubStep>(at); }
          if constexpr (kLP == 4) { lds64<n * kSubStep>(at, h[c][2 * i], h[c][2 * i + 1]); }
          if constexpr (kLP == 8) { lds128<n * kSubStep>(at, h[c][0], h[c][1], h[c][2], h[c][3]); }
        };
        if ((g0 + 4u) * kCPC <= p.pq_dim) {
          static_for<kCodes>(look_up);
        } else {
#pragma unroll
          for (uint32_t c = 0; c < 4; c++) { h[c][0] = h[c][1] = h[c][2] = h[c][3] = 0u; }
          static_for<kCodes>([&](auto nc) {
            if (g0 * kCPC + decltype(nc)::value < p.pq_dim) { look_up(nc); }
          });
        }
      }
    };
    uint32_t nxt[kNW];
#pragma unroll
    for (uint32_t i = 0; i < kNW; i++) { nxt[i] = 0u; }
    group_ref nx_g = group_of(blockIdx.x);
    load_words(nx_g, 0, nxt);
    for (uint32_t t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
      const group_ref s_g = nx_g;
      nx_g                = group_of(t + gridDim.x);
      bool counts = lane < s_g.n_rows;
      if (p.filter_bits != nullptr && counts && half == 0u) {
        const int64_t id = __ldg(p.ids + uint64_t(s_g.arena) * 32u + lane);
        counts = id >= 0 && uint64_t(id) < p.filter_nbits && ((__ldg(p.filter_bits + (id >> 5)) >> (id & 31)) & 1u);
      }
      const bool in = s_g.n_rows != 0u;
      float rn0 = 0.0f, rn1 = 0.0f;
      for (uint32_t kb = 0; kb < n_blocks; kb++) {
        uint32_t w[kNW], h[4][4];
#pragma unroll
        for (uint32_t i = 0; i < kNW; i++) { w[i] = nxt[i]; }
        if (kb + 1 < n_blocks) {
          load_words(s_g, kb + 1, nxt);
        } else {
          load_words(nx_g, 0, nxt);
        }
        look(s_g, kb, w, h);
        if (in && !p.is_ip) {
#pragma unroll
          for (uint32_t c = 0; c < 4; c++) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
              rn0 = fma_half_sq(h[c][i], false, rn0);
              rn1 = fma_half_sq(h[c][i], true, rn1);
            }
          }
        }
        // (a lane whose wait runs out goes through the tile's blocks without another one, so that the warp stays together)
        if (ok) { ok = mbar_wait(bar_empty + stage * 8, phase ^ 1u, p.spin_limit); }
        if (in) {
          const uint32_t dst = base_a + stage * kStage + kABytes;
#pragma unroll
          for (uint32_t c = 0; c < 4; c++) {
            const uint32_t g = kb * 8u + half * 4u + c;
            if (g < p.k_chunks && g != p.data_chunks) { sts128(dst + swz(r, half * 4u + c), h[c][0], h[c][1], h[c][2], h[c][3]); }
          }
          if (kb + 1 == n_blocks) {
            // the extra chunk: each thread of a row its half of |r|^2 in two halfs, the first one the mask
            const float rn    = rn0 + rn1;
            const float hi    = __half2float(__float2half_rn(rn));
            const uint32_t at = dst + swz(r, p.data_chunks & 7u) + half * 8u;
            sts64(at, half2_bits(hi, rn - hi), half2_bits(counts || half != 0u ? 0.0f : kMaskHalf, 0.0f));
          }
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) { mbar_arrive(bar_full + stage * 8); }
        if (++stage == p.n_stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (__any_sync(kFullMask, !ok)) {
        ok = false;
        break;
      }
    }
  } else if (warp == kTmaWarp) {
    // ---------------- queries of the list -> operand A ----------------
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      for (uint32_t t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
        const uint2 d = __ldg(reinterpret_cast<const uint2*>(p.tiles + t));  // first pair, pairs
        // rows of the box: what follows the tile's own pairs is another tile's and goes unused
        const CUtensorMap* map = d.y <= 16u ? &map_16 : (d.y <= 64u ? &map_64 : &map_128);
        const uint32_t bytes   = (d.y <= 16u ? 16u : (d.y <= 64u ? 64u : 128u)) * kBlockK * 2u;
        for (uint32_t kb = 0; kb < n_blocks; kb++) {
          if (!mbar_wait(bar_empty + stage * 8, phase ^ 1u, p.spin_limit)) {
            ok = false;
            break;
          }
          // (test only: a block that never comes, so that the wait for it runs out)
          if (kb + 1 != p.skip_kb || t != blockIdx.x) {
            mbar_arrive_expect_tx(bar_full + stage * 8, bytes);
            tma_load_2d(base_a + stage * kStage, map, bar_full + stage * 8, int(kb * kBlockK), int(d.x));
          }
          if (++stage == p.n_stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      uint32_t stage = 0, phase = 0, it = 0, nx_rows = 0;
      if (blockIdx.x < n_tiles) { nx_rows = __ldg(&p.tiles[blockIdx.x].n_groups); }
      for (uint32_t t = blockIdx.x; ok && t < n_tiles; t += gridDim.x, it++) {
        const uint32_t n = nx_rows * 32u;
        if (t + gridDim.x < n_tiles) { nx_rows = __ldg(&p.tiles[t + gridDim.x].n_groups); }
        // fp32 accumulate, half x half, both K-major, M = 128
        const uint32_t idesc = (1u << 4) | ((n >> 3) << 17) | ((kTileQ >> 4) << 24);
        const uint32_t acc   = it & 1u;
        if (!mbar_wait(bar_tempty + acc * 8, ((it >> 1) & 1u) ^ 1u, p.spin_limit)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * kTileR;
        for (uint32_t kb = 0; kb < n_blocks; kb++) {
          if (!mbar_wait(bar_full + stage * 8, phase, p.spin_limit)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa  = base_a + stage * kStage;
          const uint64_t da  = make_desc_sw128(sa), db = make_desc_sw128(sa + kABytes);
          const uint32_t nk  = min(4u, (p.k_chunks - kb * 8u) >> 1);
#pragma unroll
          for (uint32_t k = 0; k < 4; k++) {
            if (k >= nk) { break; }
            tc_mma_f16(tmem_d, da + k * 2u, db + k * 2u, idesc, (kb | k) != 0u);  // 32 bytes of K per step
          }
          tc_commit(bar_empty + stage * 8);
          if (++stage == p.n_stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) { tc_commit(bar_tfull + acc * 8); }
      }
    }
    __syncwarp();
  } else if (warp >= kEpiWarp) {
    // ---------------- epilogue: thread = query, minimum of every eight rows ----------------
    const uint32_t quarter = warp & 3u;
    const uint32_t r       = quarter * 32u + lane;
    uint32_t it            = 0;
    uint4 nx_d             = make_uint4(0u, 0u, 0u, 0u);
    float4 nx_rec          = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    uint4 nx_g             = nx_d;
    auto load_tile         = [&](uint32_t t) {
      nx_d = __ldg(reinterpret_cast<const uint4*>(p.tiles + t));
      nx_g = __ldg(reinterpret_cast<const uint4*>(&p.tiles[t].group[lane & 7u]));  // lane g: group g
      if (r < nx_d.y) { nx_rec = __ldg(p.pair_rec + nx_d.x + r); }
    };
    if (blockIdx.x < n_tiles) { load_tile(blockIdx.x); }
    for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x, it++) {
      const uint4 d0 = nx_d, dg = nx_g;
      const float mul = nx_rec.x, add = nx_rec.y;
      float4* out    = p.units + __float_as_uint(nx_rec.z);
      uint4* codes   = kCodes ? p.row_codes + __float_as_uint(nx_rec.z) : nullptr;
      const uint64_t per = dup2(nx_rec.w);
      if (t + gridDim.x < n_tiles) { load_tile(t + gridDim.x); }
      const uint32_t acc = it & 1u;
      if (ok && !mbar_wait(bar_tfull + acc * 8, (it >> 1) & 1u, p.spin_limit)) { ok = false; }
      if (__any_sync(kFullMask, !ok)) {
        ok = false;
        break;
      }
      tc_fence_after();
      if (quarter * 32u < d0.y) {
        // (masked rows give values of 2^30 in the scaled domain, a pair without bounds +inf: see rescore.cu)
        const uint32_t tm = tmem_base + ((quarter * 32u) << 16) + acc * kTileR;
        for (uint32_t g = (warp - kEpiWarp) >> 2; g < d0.z; g += kEpiWarps / 4u) {
          uint32_t x[32];
          tmem_ld32_async(tm + g * 32u, x);
          const uint32_t pr = __shfl_sync(kFullMask, dg.y, int(g)), gl = __shfl_sync(kFullMask, dg.z, int(g));
          const uint32_t p0 = (pr >> 8) & 0xFFu, np = (pr >> 16) & 0xFFu;  // the group's pairs
          tmem_ld_wait(x);
          float m[4], least[4];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            float a = min3(__uint_as_float(x[8 * u]), __uint_as_float(x[8 * u + 1]), __uint_as_float(x[8 * u + 2]));
            a       = min3(a, __uint_as_float(x[8 * u + 3]), __uint_as_float(x[8 * u + 4]));
            a       = min3(a, __uint_as_float(x[8 * u + 5]), __uint_as_float(x[8 * u + 6]));
            a       = fminf(a, __uint_as_float(x[8 * u + 7]));
            m[u]    = __fmaf_rn(a, mul, add);
            least[u] = a;
          }
          const bool mine = r - p0 < np;
          if (mine) { out[gl] = make_float4(m[0], m[1], m[2], m[3]); }
          if constexpr (kCodes) {
            // rows above it in whole steps, at most 15: the nearest integer of (steps - 1/2), which never exceeds the steps, in the
            // low bits of a float of 1.5 2^23; shifted and summed, all but those bits come to a constant
            uint32_t code[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const uint64_t low = dup2(least[u]);
              code[u]            = 0u - 0x3F400000u;
#pragma unroll
              for (int e = 0; e < 8; e += 2) {
                const uint64_t d = fma2(sub2(pack2(x[8 * u + e], x[8 * u + e + 1]), low), per, dup2(-0.5f));
                code[u] += __float_as_uint(fminf(lo2(d), 15.0f) + 12582912.0f) << (4 * e);
                code[u] += __float_as_uint(fminf(hi2(d), 15.0f) + 12582912.0f) << (4 * e + 4);
              }
            }
            if (mine) { codes[gl] = make_uint4(code[0], code[1], code[2], code[3]); }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(bar_tempty + acc * 8); }
    }
  }
  if (!ok) { atomicExch(p.error, ERR_TIMEOUT); }

  tc_fence_before();
  if (__syncthreads_or(!ok)) {
    // a time-out: give MMAs that are still in flight time to finish before their memory is released
    for (int i = 0; i < 64; i++) { __nanosleep(1000); }
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------
// work list
// ------------------------------------------------------------------------------------------------
// One warp per query: inclusive sums over its probes of list sizes and of 32-row groups; list_count[l]++ for
// every probe of a non-empty list.  A list id out of range (caller-given probes) counts as an empty list.
__global__ void count_pairs_kernel(const uint32_t* __restrict__ probes, const uint32_t* __restrict__ list_sizes,
                                   uint32_t n_lists, uint32_t n_queries, uint32_t n_probes,
                                   uint32_t* __restrict__ chunk_index, uint32_t* __restrict__ group_index,
                                   uint32_t* __restrict__ list_count)
{
  chain_begin();
  const uint32_t q    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (q >= n_queries) { return; }
  uint32_t carry = 0, gcarry = 0;
  for (uint32_t p0 = 0; p0 < n_probes; p0 += 32) {
    const uint32_t p = p0 + lane;
    uint32_t v       = 0;
    if (p < n_probes) {
      const uint32_t label = probes[size_t(q) * n_probes + p];
      v                    = label < n_lists ? list_sizes[label] : 0u;
      if (v > 0) { atomicAdd(list_count + label, 1u); }
    }
    uint32_t g = (v + 31u) >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(kFullMask, v, d), u = __shfl_up_sync(kFullMask, g, d);
      if (lane >= uint32_t(d)) {
        v += t;
        g += u;
      }
    }
    if (p < n_probes) {
      chunk_index[size_t(q) * n_probes + p] = carry + v;
      group_index[size_t(q) * n_probes + p] = gcarry + g;
    }
    carry += __shfl_sync(kFullMask, v, 31);
    gcarry += __shfl_sync(kFullMask, g, 31);
  }
}

// Blocks of 64 lists: where a list's pairs and tiles go (one atomic per block and kind; the order of the blocks
// does not matter), the tiles themselves, and list_count[l] becomes the list's cursor for the operand kernel.
// Lists of at most kPackPairs pairs share tiles: their groups form one stream that is cut every eight (eight
// lists' pairs still fit a tile).  A list with more pairs has tiles of its own, its queries dealt evenly over
// tiles of at most 128.  The block's pairs are ordered accordingly: first the sharing lists'.
constexpr uint32_t kPackPairs   = kTileQ / 8;
// 64 lists per block share tiles better, 16 give more blocks: 16 below 32,768 lists.  A whole call of 10,000 queries x 20
// probes over 3 M rows, 16 / 64 lists per block (us): 1,000 lists 1,029 / 1,073, 4,000 642 / 649, 9,000 684 / 685, 16,000
// 771 / 772, 24,000 711 / 707, 32,000 766 / 762, 50,000 920 / 912.  (The kernel alone, 4,000 lists of 1,000 rows and 64
// probes: 50 / 111.)
template <uint32_t kListsPerBlock>
__global__ void __launch_bounds__(256)
make_tiles_kernel(uint32_t* __restrict__ list_count, const uint32_t* __restrict__ list_sizes,
                  const uint64_t* __restrict__ row_off, uint32_t n_lists, filter_tile* __restrict__ tiles,
                  uint32_t* __restrict__ counters)
{
  chain_begin();
  // exclusive sums over the block's lists: pairs and groups of sharing lists, pairs and tiles of the others
  constexpr uint32_t kScan = kListsPerBlock < 32u ? 32u : kListsPerBlock;
  __shared__ uint32_t s_off[4][kScan + 1], s_count[kScan], s_size[kScan], s_arena[kScan], s_warp[4], s_base[2];
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  const uint32_t l   = blockIdx.x * kListsPerBlock + tid;
  uint32_t v[4] = {0u, 0u, 0u, 0u}, x[4];
  if (tid < kScan) {
    const uint32_t c    = tid < kListsPerBlock && l < n_lists ? list_count[l] : 0u;
    const uint32_t size = c > 0 ? list_sizes[l] : 0u, ng = (size + 31u) >> 5;
    const bool share    = c <= kPackPairs;
    v[share ? 0 : 2]    = c;
    v[share ? 1 : 3]    = share ? ng : ceildiv(c, kTileQ) * ceildiv(ng, 8u);
    s_count[tid]        = c;
    s_size[tid]         = size;
    s_arena[tid]        = c > 0 ? uint32_t(row_off[l] >> 5) : 0u;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      x[k] = v[k];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(kFullMask, x[k], d);
        if (lane >= uint32_t(d)) { x[k] += o; }
      }
      if (tid == 31) { s_warp[k] = x[k]; }
    }
  }
  __syncthreads();
  if (tid < kListsPerBlock) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t inc = x[k] + (tid >= 32u ? s_warp[k] : 0u);
      s_off[k][tid]      = inc - v[k];
      if (tid == kListsPerBlock - 1) { s_off[k][kListsPerBlock] = inc; }
    }
  }
  __syncthreads();
  const uint32_t n_groups = s_off[1][kListsPerBlock], n_own = s_off[3][kListsPerBlock];
  const uint32_t n_shared = (n_groups + 7u) >> 3;  // tiles of the sharing lists
  if (tid == 0) {
    const uint32_t np = s_off[0][kListsPerBlock] + s_off[2][kListsPerBlock], nt = n_shared + n_own;
    s_base[0]         = np ? atomicAdd(counters, np) : 0u;
    s_base[1]         = nt ? atomicAdd(counters + 1, nt) : 0u;
  }
  __syncthreads();
  // first pair of a list
  auto pair0 = [&](uint32_t i) {
    return s_base[0] + (s_count[i] <= kPackPairs ? s_off[0][i] : s_off[0][kListsPerBlock] + s_off[2][i]);
  };
  if (tid < kListsPerBlock && l < n_lists) { list_count[l] = pair0(tid); }
  auto find = [&](const uint32_t* off, uint32_t y) {  // last list whose first element is <= y
    uint32_t lo = 0, hi = kListsPerBlock - 1;
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (off[mid] <= y) {
        lo = mid;
      } else {
        hi = mid - 1;
      }
    }
    return lo;
  };
  // {arena group; rows, first pair, pairs as bytes; group of the list; -}
  auto group_of = [&](uint32_t i, uint32_t g, uint32_t p0, uint32_t np) {
    return make_uint4(s_arena[i] + g, min(32u, s_size[i] - g * 32u) | (p0 << 8) | (np << 16), g, 0u);
  };
  for (uint32_t y = tid; y < n_shared * 8u; y += 256) {
    uint4* t             = reinterpret_cast<uint4*>(tiles + s_base[1] + (y >> 3));
    const uint32_t first = find(s_off[1], y & ~7u);
    if (y < n_groups) {
      const uint32_t i = find(s_off[1], y);
      t[1 + (y & 7u)]  = group_of(i, y - s_off[1][i], s_off[0][i] - s_off[0][first], s_count[i]);
    }
    if ((y & 7u) == 0u) {
      const uint32_t end  = min(y + 8u, n_groups);
      const uint32_t last = find(s_off[1], end - 1u);
      t[0] = make_uint4(pair0(first), s_off[0][last] + s_count[last] - s_off[0][first], end - y, 0u);
    }
  }
  for (uint32_t y = tid; y < n_own * 8u; y += 256) {
    const uint32_t i = find(s_off[3], y >> 3), k = (y >> 3) - s_off[3][i];
    uint4* t         = reinterpret_cast<uint4*>(tiles + s_base[1] + n_shared + (y >> 3));
    const uint32_t groups = (s_size[i] + 31u) >> 5, cnt = s_count[i];
    const uint32_t nrt = ceildiv(groups, 8u), mt = k / nrt, rt = k - mt * nrt, nmt = ceildiv(cnt, kTileQ);
    const uint32_t q0 = uint32_t(uint64_t(cnt) * mt / nmt), q1 = uint32_t(uint64_t(cnt) * (mt + 1) / nmt);
    const uint32_t g  = rt * 8u + (y & 7u);
    if (g < groups) { t[1 + (y & 7u)] = group_of(i, g, 0u, q1 - q0); }
    if ((y & 7u) == 0u) { t[0] = make_uint4(pair0(i) + q0, q1 - q0, min(8u, groups - rt * 8u), 0u); }
  }
}

// The query operand: sixteen lanes per (query, probe) pair.  `cursor`: next place of every list's pairs, which orders the
// pairs by list.  A pair of an empty list has none.
// Row of the operand: L2 -2 (q - c) s, inner product -q s_q, in half precision, then 1, 1, mask, 0, 1, 1, 0, 0
// against the row side's |r|^2 and mask.  Record: {factor, constant, first group of the pair's bounds, steps per value}.
__global__ void __launch_bounds__(256)
pair_operands_kernel(const operand_params p, const uint32_t* __restrict__ probes, const uint32_t* __restrict__ list_sizes,
                     uint32_t n_lists, const uint32_t* __restrict__ group_index, uint32_t n_pairs, uint32_t n_probes,
                     uint32_t max_groups, uint32_t* __restrict__ cursor, __half* __restrict__ operand,
                     float4* __restrict__ pair_rec, float* __restrict__ pair_norm)
{
  chain_begin();
  const uint32_t i    = (blockIdx.x * 256u + threadIdx.x) >> 4;
  const uint32_t lane = threadIdx.x & 15u;
  const unsigned half_mask = 0xFFFFu << (threadIdx.x & 16u);
  if (i >= n_pairs) { return; }
  const uint32_t label = __ldg(probes + i);
  if (label >= n_lists || __ldg(list_sizes + label) == 0) { return; }
  const uint32_t q = i / n_probes, pi = i - q * n_probes;
  uint32_t pos     = 0;
  if (lane == 0) { pos = atomicAdd(cursor + label, 1u); }
  pos = __shfl_sync(half_mask, pos, 0, 16);
  const float* qr = p.rot_q + size_t(q) * p.rot_dim;
  const float* cr = p.centers + size_t(label) * p.rot_dim;
  const float sq  = p.is_ip ? __ldg(p.q_scale + q) : p.scale;
  uint4* out      = reinterpret_cast<uint4*>(operand + size_t(pos) * (p.k_chunks * 8u));
  float a_sum = 0.0f, b_sum = 0.0f;  // L2: |d|^2 of the rounded difference, largest |d_i|; inner product: |c|^2, q.c
  for (uint32_t g = lane; g < p.k_chunks; g += 16) {
    uint32_t h[4] = {0u, 0u, 0u, 0u};
    if (g < p.data_chunks) {
      float qv[8], cv[8];
      if (p.vec_rows) {
        const float4 a0 = __ldg(reinterpret_cast<const float4*>(qr + g * 8u));
        const float4 a1 = __ldg(reinterpret_cast<const float4*>(qr + g * 8u) + 1);
        const float4 b0 = __ldg(reinterpret_cast<const float4*>(cr + g * 8u));
        const float4 b1 = __ldg(reinterpret_cast<const float4*>(cr + g * 8u) + 1);
        qv[0] = a0.x; qv[1] = a0.y; qv[2] = a0.z; qv[3] = a0.w;
        qv[4] = a1.x; qv[5] = a1.y; qv[6] = a1.z; qv[7] = a1.w;
        cv[0] = b0.x; cv[1] = b0.y; cv[2] = b0.z; cv[3] = b0.w;
        cv[4] = b1.x; cv[5] = b1.y; cv[6] = b1.z; cv[7] = b1.w;
      } else {
#pragma unroll
        for (uint32_t e = 0; e < 8; e++) {
          const uint32_t k  = g * 8u + e;
          const uint32_t js = k / p.len_pad, kk = k - js * p.len_pad;
          const bool in     = js < p.pq_dim && kk < p.pq_len;
          qv[e]             = in ? __ldg(qr + js * p.pq_len + kk) : 0.0f;
          cv[e]             = in ? __ldg(cr + js * p.pq_len + kk) : 0.0f;
        }
      }
#pragma unroll
      for (int e = 0; e < 4; e++) {
        float a = qv[2 * e], b = qv[2 * e + 1];
        if (!p.is_ip) {
          a     = __fsub_rn(a, cv[2 * e]);
          b     = __fsub_rn(b, cv[2 * e + 1]);
          b_sum = fmaxf(b_sum, fmaxf(fabsf(a), fabsf(b)));
        } else {
          b_sum = __fmaf_rn(a, cv[2 * e], b_sum);
          b_sum = __fmaf_rn(b, cv[2 * e + 1], b_sum);
          a_sum = __fmaf_rn(cv[2 * e], cv[2 * e], a_sum);
          a_sum = __fmaf_rn(cv[2 * e + 1], cv[2 * e + 1], a_sum);
        }
        const __half2 v = __floats2half2_rn(a * sq, b * sq);
        const float2 f  = __half22float2(v);
        if (!p.is_ip) {
          a_sum = __fmaf_rn(f.x, f.x, a_sum);
          a_sum = __fmaf_rn(f.y, f.y, a_sum);
          h[e]  = half2_bits(-2.0f * f.x, -2.0f * f.y);
        } else {
          h[e] = half2_bits(-f.x, -f.y);
        }
      }
    } else if (g == p.data_chunks) {
      h[0] = half2_bits(1.0f, 1.0f);
      h[1] = half2_bits(kMaskHalf, 0.0f);
      h[2] = half2_bits(1.0f, 1.0f);
    }
    out[g] = make_uint4(h[0], h[1], h[2], h[3]);
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    a_sum += __shfl_xor_sync(half_mask, a_sum, o);
    const float x = __shfl_xor_sync(half_mask, b_sum, o);
    b_sum         = p.is_ip ? b_sum + x : fmaxf(b_sum, x);
  }
  if (lane == 0) {
    float mul, add, norm, per;
    if (p.is_ip) {
      mul  = 1.0f / (sq * p.scale);
      add  = -b_sum;
      norm = sqrtf(a_sum) * 1.00001f;
      per  = mul * sq / p.row_step;
    } else {
      mul  = p.inv_scale2;
      add  = a_sum * p.inv_scale2;
      norm = sqrtf(add) * 1.00001f;
      const float far = b_sum + p.rcomp_max;
      per  = mul / (p.row_step * add);
      // differences that do not fit half precision: no bound for this pair
      if (!(b_sum * p.scale <= 16384.0f)) { add = INFINITY; }
      if (!(float(p.pq_len) * far * far < p.entry_limit)) { norm = -norm - 1e-30f; }
    }
    // (no steps that make sense: every row counts as its unit)
    if (!(per > 0.0f && per < 1e25f && add < INFINITY)) { per = 0.0f; }
    pair_rec[pos] = make_float4(mul, add, __uint_as_float(q * max_groups + (pi > 0 ? __ldg(group_index + i - 1) : 0u)),
                                per * 0.9999f);
    pair_norm[i]  = norm;
  }
}

// Inner product: the power of two that brings a query's norm near 64.  One warp per query.
__global__ void query_scale_kernel(const float* __restrict__ rot_q, uint32_t n_queries, uint32_t rot_dim,
                                   float* __restrict__ q_scale)
{
  chain_begin();
  const uint32_t q    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (q >= n_queries) { return; }
  float ss = 0.0f;
  for (uint32_t i = lane; i < rot_dim; i += 32) {
    const float v = rot_q[size_t(q) * rot_dim + i];
    ss            = __fmaf_rn(v, v, ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { ss += __shfl_xor_sync(kFullMask, ss, o); }
  if (lane == 0) {
    const int e = int((__float_as_uint(ss) >> 23) & 0xFFu) - 127;  // ss in [2^e, 2^(e+1))
    const int h = min(100, max(-100, 6 - (e >> 1) - (e & 1)));
    q_scale[q]  = ss > 0.0f && ss < INFINITY ? __uint_as_float(uint32_t(127 + h) << 23) : 1.0f;
  }
}

// ------------------------------------------------------------------------------------------------
// half-precision codebooks
// ------------------------------------------------------------------------------------------------
__global__ void book_stats_kernel(const float* __restrict__ pq, uint32_t len, uint32_t book, float* __restrict__ tmp)
{
  // one block per subspace: largest squared norm of a codeword, largest |component|
  __shared__ float s_a[8], s_b[8];
  const float* c = pq + size_t(blockIdx.x) * len * book;
  float a = 0.0f, b = 0.0f;
  for (uint32_t e = threadIdx.x; e < book; e += blockDim.x) {
    float ss = 0.0f;
    for (uint32_t k = 0; k < len; k++) {
      const float v = c[size_t(k) * book + e];
      ss            = __fmaf_rn(v, v, ss);
      b             = fmaxf(b, fabsf(v));
    }
    a = fmaxf(a, ss);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    a = fmaxf(a, __shfl_xor_sync(kFullMask, a, d));
    b = fmaxf(b, __shfl_xor_sync(kFullMask, b, d));
  }
  if ((threadIdx.x & 31u) == 0) {
    s_a[threadIdx.x >> 5] = a;
    s_b[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < (blockDim.x >> 5); w++) {
      a = fmaxf(a, s_a[w]);
      b = fmaxf(b, s_b[w]);
    }
    tmp[2 * blockIdx.x]     = a;
    tmp[2 * blockIdx.x + 1] = b;
  }
}
__global__ void book_scale_kernel(const float* __restrict__ tmp, uint32_t pq_dim, float* __restrict__ stats)
{
  float a = 0.0f, b = 0.0f;
  for (uint32_t j = 0; j < pq_dim; j++) {
    a += tmp[2 * j];
    b = fmaxf(b, tmp[2 * j + 1]);
  }
  a *= 1.00001f;
  // a power of two s with a * s^2 in (2^12, 2^14]: |r|^2 fits half precision, components keep their bits
  float s = 1.0f;
  if (a > 1e-30f && a < 1e30f) {
    const int e = int((__float_as_uint(a) >> 23) & 0xFFu) - 127;  // a in [2^e, 2^(e+1))
    const int h = (13 - e) >> 1;                                 // 2h + e + 1 <= 14
    s           = __uint_as_float(uint32_t(127 + h) << 23);
  }
  stats[0] = a;
  stats[1] = b;
  stats[2] = s;
}
__global__ void book_image_kernel(const float* __restrict__ pq, uint32_t len, uint32_t len_pad, uint32_t book,
                                  const float* __restrict__ stats, __half* __restrict__ out, uint32_t n)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;  // (subspace * book + entry) * len_pad + component
  if (i >= n) { return; }
  const uint32_t kk = i % len_pad, e = (i / len_pad) % book, j = i / len_pad / book;
  out[i] = __float2half_rn(kk < len ? pq[(size_t(j) * len + kk) * book + e] * stats[2] : 0.0f);
}

}  // namespace

void make_filter_book(const float* pq_centers, uint32_t pq_dim, uint32_t pq_len, uint32_t len_pad, uint32_t book,
                      __half* out, float* d_stats, float* d_tmp, cudaStream_t stream)
{
  book_stats_kernel<<<pq_dim, 256, 0, stream>>>(pq_centers, pq_len, book, d_tmp);
  book_scale_kernel<<<1, 1, 0, stream>>>(d_tmp, pq_dim, d_stats);
  const uint32_t n = pq_dim * book * len_pad;
  book_image_kernel<<<ceildiv(n, 256u), 256, 0, stream>>>(pq_centers, pq_len, len_pad, book, d_stats, out, n);
  CUDA_TRY(cudaGetLastError());
}

void launch_count_pairs(const uint32_t* probes, const uint32_t* list_sizes, uint32_t n_lists, uint32_t n_queries,
                        uint32_t n_probes, uint32_t* chunk_index, uint32_t* group_index, uint32_t* list_count,
                        cudaStream_t stream)
{
  launch_chained(count_pairs_kernel, ceildiv<uint32_t>(n_queries * 32, 256), 256, 0, stream, probes, list_sizes,
                 n_lists, n_queries, n_probes, chunk_index, group_index, list_count);
  CUDA_TRY(cudaGetLastError());
}

void launch_tiles(const uint32_t* list_sizes, const uint64_t* row_off, uint32_t n_lists, uint32_t* list_count,
                  filter_tile* tiles, uint32_t* counters, cudaStream_t stream)
{
  if (n_lists >= 32768) {
    launch_chained(make_tiles_kernel<64>, ceildiv(n_lists, 64u), 256, 0, stream, list_count, list_sizes, row_off,
                   n_lists, tiles, counters);
  } else {
    launch_chained(make_tiles_kernel<16>, ceildiv(n_lists, 16u), 256, 0, stream, list_count, list_sizes, row_off,
                   n_lists, tiles, counters);
  }
  CUDA_TRY(cudaGetLastError());
}

void launch_pair_operands(const operand_params& p, const uint32_t* probes, const uint32_t* list_sizes, uint32_t n_lists,
                          const uint32_t* group_index, uint32_t n_pairs, uint32_t n_probes, uint32_t max_groups,
                          uint32_t* cursor, __half* operand, float4* pair_rec, float* pair_norm, cudaStream_t stream)
{
  launch_chained(pair_operands_kernel, ceildiv(n_pairs, 16u), 256, 0, stream, p, probes, list_sizes, n_lists,
                 group_index, n_pairs, n_probes, max_groups, cursor, operand, pair_rec, pair_norm);
  CUDA_TRY(cudaGetLastError());
}

void launch_query_scale(const float* rot_q, uint32_t n_queries, uint32_t rot_dim, float* q_scale, cudaStream_t stream)
{
  launch_chained(query_scale_kernel, ceildiv<uint32_t>(n_queries * 32, 256), 256, 0, stream, rot_q, n_queries, rot_dim,
                 q_scale);
  CUDA_TRY(cudaGetLastError());
}

uint64_t max_filter_tiles(const index<int64_t>& idx, uint32_t n_queries, uint32_t n_probes, bool distinct)
{
  const uint64_t n_pairs = uint64_t(n_queries) * n_probes;
  // every list once (row tiles of the whole index), and the extra query groups: one more per 128 pairs of a list
  const uint64_t all     = uint64_t(idx.total_rows_padded()) / kTileR + idx.n_lists();
  const uint64_t longest = ceildiv<uint64_t>(uint64_t(idx.accum_sorted_sizes()[1]), kTileR);
  uint64_t tiles         = std::min(n_pairs * longest, all + (n_pairs / kTileQ) * longest);
  if (distinct) {
    // a list has at most n_queries pairs: at worst all of them in the n_probes longest lists
    const uint64_t probed = uint64_t(idx.accum_sorted_sizes()[n_probes]) / kTileR + n_probes;
    tiles                 = std::min(tiles, all + ceildiv<uint64_t>(n_queries, kTileQ) * probed);
  }
  return tiles;
}

void launch_filter(const filter_params& p, const __half* operand, uint32_t n_pairs, int grid, size_t smem,
                   cudaStream_t stream)
{
  const uint64_t k       = uint64_t(p.k_chunks) * 8;
  const CUtensorMap m16  = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, operand, n_pairs, k, 16, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
  const CUtensorMap m64  = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, operand, n_pairs, k, 64, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
  const CUtensorMap m128 = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, operand, n_pairs, k, 128, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
  auto go = [&](auto with_codes, auto without) {
    auto kernel = p.row_codes != nullptr ? with_codes : without;
    ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    launch_chained(kernel, grid, kFilterThreads, smem, stream, m16, m64, m128, p);
    CUDA_TRY(cudaGetLastError());
  };
  auto by_len = [&](auto bits, auto words) {
    constexpr int kB     = decltype(bits)::value;
    constexpr bool kWord = decltype(words)::value;
    switch (p.len_pad) {
      case 1: go(filter_kernel<kB, 1, kWord, true>, filter_kernel<kB, 1, kWord, false>); break;
      case 2: go(filter_kernel<kB, 2, kWord, true>, filter_kernel<kB, 2, kWord, false>); break;
      case 4: go(filter_kernel<kB, 4, kWord, true>, filter_kernel<kB, 4, kWord, false>); break;
      default: go(filter_kernel<kB, 8, kWord, true>, filter_kernel<kB, 8, kWord, false>);
    }
  };
  using std::integral_constant;
  switch (p.pq_bits) {
    case 8:
      if (p.len_pad <= 8) {
        by_len(integral_constant<int, 8>{}, std::true_type{});
      } else {
        go(filter_kernel<8, 8, false, true>, filter_kernel<8, 8, false, false>);
      }
      break;
    case 7: by_len(integral_constant<int, 7>{}, std::false_type{}); break;
    case 6: by_len(integral_constant<int, 6>{}, std::false_type{}); break;
    case 5: by_len(integral_constant<int, 5>{}, std::false_type{}); break;
    default:
      if (p.len_pad <= 8) {
        by_len(integral_constant<int, 4>{}, std::true_type{});
      } else {
        go(filter_kernel<4, 8, false, true>, filter_kernel<4, 8, false, false>);
      }
  }
}

}  // namespace cuvs::neighbors::ivf_pq
