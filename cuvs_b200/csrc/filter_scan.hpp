// Fine search in two steps (filter_scan.cu, rescore.cu): a tensor-core pass over the probed lists bounds
// every row's score from below, eight rows at a time; the rows that the bounds cannot rule out are then
// scored exactly and the k best of a query selected.  Declarations shared by the two files and search.cu.
#pragma once

#include "ivf_pq.hpp"

namespace cuvs::neighbors::ivf_pq {

constexpr uint32_t kUnitRows = 8;  // rows of a list that share one bound ("unit"); four units = one 32-row group

// One tile of the filter kernel's work: up to eight 32-row groups of lists against up to 128 (query, list) pairs
// that are consecutive in the order by list.  Group g holds rows of one list and counts for the tile's pairs
// [pair0, pair0 + n_pairs) only.
struct filter_group {
  uint32_t arena;                // first row / 32 in the arenas
  uint8_t n_rows, pair0, n_pairs, pad;
  uint32_t in_list;              // number of the group in its list
  uint32_t pad2;
};
struct filter_tile {
  uint32_t first_pair, n_pairs, n_groups, pad;
  filter_group group[8];
};

// Half-precision image of the codebooks, made once per model (index<int64_t>::filter_model).
// K layout: subspace j occupies `len_pad` consecutive halfs, entries padded with zeros.
struct operand_params {
  const float* rot_q;    // [n_q, rot_dim]
  const float* centers;  // [n_lists, rot_dim]
  const float* q_scale;  // inner product: power of two per query (launch_query_scale)
  uint32_t pq_dim, pq_len, rot_dim;
  uint32_t len_pad, data_chunks, k_chunks;  // 16-byte chunks (8 halfs) of data, and of a whole row
  int vec_rows;                             // rows of rot_q / centers are 16-byte aligned and need no padding
  int is_ip;
  float scale, inv_scale2;                  // power of two s: codewords and differences are multiplied by it
  float entry_limit, rcomp_max;             // a table entry that may exceed the limit flags its pair
  float row_step;                           // see row_step of rescore_params
};

struct filter_params {
  const __half* book;    // [pq_dim][book][len_pad]
  const uint8_t* codes;
  const int64_t* ids;
  const uint32_t* filter_bits;
  uint64_t filter_nbits;
  uint32_t book_bytes, book_size;
  uint32_t pq_dim, pq_bits, n_pieces;
  uint32_t len_pad, data_chunks, k_chunks;
  int is_ip;
  const filter_tile* tiles;
  const uint32_t* n_tiles;
  const float4* pair_rec;  // per pair, in the operand's order: {factor, constant, first group of its units, row codes per value}
  float4* units;           // [n_q, max_groups] bounds of the four units of a 32-row group
  uint4* row_codes;        // optional: [n_q, max_groups] how far above it its rows are, four bits each, in steps (row_step)
  uint32_t n_stages;
  uint32_t* error;
  uint32_t spin_limit, skip_kb;  // tc_wait_limits
};

struct rescore_params {
  const float* rot_q;
  const float* centers;  // [n_lists, rot_dim]
  const float* pq_centers;
  const uint8_t* codes;
  const int64_t* ids;
  const uint64_t* row_off;
  const uint32_t* probes;       // [n_q, n_probes]
  const uint32_t* chunk_index;  // [n_q, n_probes] inclusive sums of list sizes
  const uint32_t* group_index;  // [n_q, n_probes] inclusive sums of 32-row groups
  const float4* units;
  const uint4* row_codes;       // optional
  const float* pair_norm;
  const float* q_scale;         // inner product
  const uint32_t* error;
  uint32_t* timeouts;           // pinned host word: batches with the error word set
  const uint32_t* filter_bits;
  uint64_t filter_nbits;
  uint32_t n_lists, n_queries, n_probes, k, max_groups;
  uint32_t pq_dim, pq_len, pq_bits, rot_dim, n_pieces, book_size;
  // shared-memory plan; book_bytes 0: the codebook stays in global memory
  uint32_t groups, group_threads, group_bytes, book_bytes, cap, list_cap;
  int cosine, metric;
  float post_scale;
  // error model (see rescore.cu)
  float e1, kappa, e0, e2, delta_lo, delta_hi, eta, sum_limit, rmax, ip_gemm, ip_lut;
  // step of the row codes: L2 |d|^2 row_step, inner product row_step over the query's scale (less what rounding may do)
  float row_step;
  int sharpen;    // wide bounds: score what is certainly wanted first
  int saturates;  // the table type saturates (8-bit tables)
  uint32_t* claim;  // zero on entry: next query to take
  int64_t* neighbors;
  float* distances;
};

struct filter_plan {
  bool use = false;
  uint32_t n_stages = 0;
  size_t filter_smem = 0;
  uint32_t groups = 0, group_threads = 0, group_bytes = 0, book_bytes = 0, cap = 0, list_cap = 0;
  size_t rescore_smem = 0;
};

// Whether (and with which shared-memory plan) a search runs on the two-step path (k <= 128).
filter_plan plan_filter(const raft::resources& res, const index<int64_t>& idx, int lut_kind, bool out_half, bool is_ip,
                        uint32_t k, uint32_t n_probes, uint32_t n_queries, bool row_codes);

// `operand`: [n_pairs, k_chunks * 8] halfs written by launch_pair_operands.
void launch_filter(const filter_params& p, const __half* operand, uint32_t n_pairs, int grid, size_t smem,
                   cudaStream_t stream);
void launch_rescore(const rescore_params& p, int lut_kind, bool out_half, bool is_ip, int grid, size_t smem,
                    cudaStream_t stream);

// Sample offsets, group offsets and the histogram of pairs per list.
void launch_count_pairs(const uint32_t* probes, const uint32_t* list_sizes, uint32_t n_lists, uint32_t n_queries,
                        uint32_t n_probes, uint32_t* chunk_index, uint32_t* group_index, uint32_t* list_count,
                        cudaStream_t stream);
// Tiles, and list_count becomes every list's cursor into the pairs ordered by list; counters: [0] pairs,
// [1] tiles (zero on entry).
void launch_tiles(const uint32_t* list_sizes, const uint64_t* row_off, uint32_t n_lists, uint32_t* list_count,
                  filter_tile* tiles, uint32_t* counters, cudaStream_t stream);
// The query operand of every pair, at the pair's place (`cursor`: the next one of every list), its record, and
// pair_norm [n_q * n_probes]: |q - c| (L2; negative: flagged) or |c| (inner product).
void launch_pair_operands(const operand_params& p, const uint32_t* probes, const uint32_t* list_sizes, uint32_t n_lists,
                          const uint32_t* group_index, uint32_t n_pairs, uint32_t n_probes, uint32_t max_groups,
                          uint32_t* cursor, __half* operand, float4* pair_rec, float* pair_norm, cudaStream_t stream);
void launch_query_scale(const float* rot_q, uint32_t n_queries, uint32_t rot_dim, float* q_scale, cudaStream_t stream);
// Upper bound on the number of tiles; `distinct`: no query probes a list twice (caller-given probes may).
uint64_t max_filter_tiles(const index<int64_t>& idx, uint32_t n_queries, uint32_t n_probes, bool distinct);

// Half-precision codebooks: `out` [pq_dim][book][len_pad], stats[0] = sum over subspaces of the largest squared
// codeword norm, stats[1] = largest |component|, both of the fp32 codebook; `scale_out` the power of two.
void make_filter_book(const float* pq_centers, uint32_t pq_dim, uint32_t pq_len, uint32_t len_pad, uint32_t book,
                      __half* out, float* d_stats /* [3]: ss, max, scale */, float* d_tmp /* [2 * pq_dim] */,
                      cudaStream_t stream);

}  // namespace cuvs::neighbors::ivf_pq
