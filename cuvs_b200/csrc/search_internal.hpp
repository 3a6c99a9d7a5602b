// Declarations shared between the search translation units.
#pragma once

#include "ivf_pq.hpp"

#include <cuda.h>

namespace cuvs::neighbors::ivf_pq {

#ifdef __CUDACC__
// Score -> reported distance (postprocess_distances, cpp/src/neighbors/ivf_common.cuh:175-252).
__device__ __forceinline__ float postprocess_distance(float score, int metric, float scale)
{
  switch (metric) {
    case 0: return scale != 1.0f ? __fmul_rn(score, __fmul_rn(scale, scale)) : score;
    case 1: return scale != 1.0f ? __fmul_rn(__fsqrt_rn(score), scale) : __fsqrt_rn(score);
    case 6: return __fmul_rn(score, __fmul_rn(__fmul_rn(-1.0f, scale), scale));
    default: {
      const float f = __fmul_rn(scale, scale);
      return f != 1.0f ? __fmul_rn(score, f) : score;
    }
  }
}
#endif

struct scan_plan {
  uint32_t n_groups, group_threads, pqc_in_smem, pqc_bytes, group_bytes, lut_bytes, base_bytes,
    merge_bytes, tmem_cols, tmem_slot_off, lut_global, base_double;
  size_t total_bytes;
};
scan_plan plan_scan(const raft::resources& res, const index<int64_t>& idx, int lut_kind, bool is_ip,
                    uint32_t k);

// Coarse stage (coarse.cu): for every query the n_probes lists with the smallest
//   score[q, l] = alpha * sum_k centers[l, k] * fq[q, k]
// sorted by (score, list id) ascending.  `scores_out` (optional) receives the selected scores.
// `half_scores`: every score is rounded to half precision before the selection (fp16 coarse search).
size_t coarse_workspace_bytes(uint32_t n_queries, uint32_t n_lists, uint32_t n_probes);
void select_clusters(raft::resources& res, const float* centers, uint32_t n_lists, uint32_t dim_ext,
                     float alpha, const float* fq, uint32_t n_queries, uint32_t n_probes,
                     uint32_t* probes, float* scores_out, void* workspace, size_t workspace_bytes,
                     bool half_scores = false);

// Per row the k smallest (value, position), ascending (k <= 4096).  `row_ends` (optional): row r holds only
// row_ends[(r + 1) * ends_stride - 1] values; results beyond them have a NaN score.
void select_rows(raft::resources& res, const float* rows, uint32_t n_rows, uint32_t row_len, uint32_t k,
                 uint32_t* out_idx, float* out_scores, const uint32_t* row_ends = nullptr, uint32_t ends_stride = 0);

// Tensor-core coarse stage (coarse_tc.cu): same contract and bit-identical probes as
// select_clusters; `centers_hi/lo` are the TF32 split of `centers`, `cmax` the largest row norm.
// `exact_operands`: every operand is exact in TF32 and every partial sum in fp32 (small integers):
// one product per K step, and the guard allows for no split error.
// TMA descriptor of a row-major [rows, cols] matrix, box [box_rows, box_cols], zero fill outside (coarse_tc.cu).
CUtensorMap make_map_2d(CUtensorMapDataType type, uint32_t elem_bytes, const void* ptr, uint64_t rows, uint64_t cols,
                        uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swizzle);
bool coarse_tc_usable(uint32_t n_lists, uint32_t n_probes, uint32_t dim_ext);
size_t coarse_tc_workspace_bytes(uint32_t n_queries, uint32_t n_lists, uint32_t dim_ext);
// Prepares `hi` / `lo` (TF32 split of the centre rows) with column `ext_col` (the |c|^2 column of L2
// metrics; >= dim_ext: none) divided by a power of two `ext_scale` close to the largest |c|, and `cmax`,
// the largest norm of a row so prepared; select_clusters_tc is given the same ext_col / ext_scale and
// multiplies the queries' entry of that column by it.  Synchronises the stream.
void prepare_tc_centers(cudaStream_t stream, const float* centers, uint32_t n_lists, uint32_t dim_ext,
                        uint32_t ext_col, float* hi, float* lo, float* cmax, float* ext_scale);
void select_clusters_tc(raft::resources& res, const float* centers, const float* centers_hi,
                        const float* centers_lo, float cmax, uint32_t n_lists, uint32_t dim_ext,
                        float alpha, const float* fq, uint32_t n_queries, uint32_t n_probes,
                        uint32_t* probes, float* scores_out, void* workspace, size_t workspace_bytes,
                        bool exact_operands = false, uint32_t ext_col = ~0u, float ext_scale = 1.0f);
void coarse_tc_status(raft::resources& res, const void* workspace, uint32_t n_queries, uint32_t n_lists,
                      uint32_t dim_ext, uint32_t* error, uint32_t* n_fallback);

// Probe selection alone (diagnostics / stage-wise tests): mode 0 = automatic, 1 = exact SIMT path,
// 2 = tensor-core path.  status[0] = error word, status[1] = queries redone exactly (mode 2).
void coarse_only(raft::resources& res, const index<int64_t>& idx, const void* queries, elem_t qtype,
                 uint32_t n_queries, uint32_t n_probes, int mode, uint32_t* probes, float* scores,
                 uint32_t* status);

// products of the TF32 split the tensor-core coarse GEMM issues per K step (1, 2 or 3)
void set_coarse_tc_products(int products);
// process-wide override used by tests: false = the tensor-core coarse GEMM streams both operands even
// where the query tile could stay resident in shared memory
void set_coarse_tc_resident(bool on);
// Bounded waits of the tensor-core kernels (coarse_tc.cu, filter_scan.cu, label_tc.cu): iterations a wait may take, and for
// tests 1 + index of the K block of every CTA's first tile that is never brought (0 = none).  Process-wide.
struct wait_limits {
  uint32_t spin_limit, skip_kb;
};
wait_limits tc_wait_limits();
void set_tc_wait_test(uint32_t spin_limit /* 0 = the default */, uint32_t skip_kb);
void set_coarse_mode(int mode);  // process-wide override used by tests: 0 auto, 1 SIMT, 2 tensor core
// process-wide override used by tests: 0 = the per-subspace codebook goes to tensor memory where it
// fits, 1 = never (shared memory, else global memory)
void set_scan_codebook_home(int home);

// Nearest list of every row: labels[i] = argmin_l alpha * sum_k centers[l,k] * x[i,k], ties to the
// lowest l (equals select_clusters with n_probes = 1).  `best` is scratch of n_rows * 8 bytes.
void assign_nearest(raft::resources& res, const float* centers, uint32_t n_lists, uint32_t dim_ext,
                    float alpha, const float* x_ext, uint32_t n_rows, uint32_t* labels,
                    unsigned long long* best);

// The same for the rows named in row_list[0 .. *n_listed) (both on the device), whose `best` is all ones; other labels stay as
// they are.
void assign_nearest_listed(raft::resources& res, const float* centers, uint32_t n_lists, uint32_t dim_ext, float alpha,
                           const float* x_ext, uint32_t n_rows, const uint32_t* row_list, const uint32_t* n_listed,
                           uint32_t* labels, unsigned long long* best);
// out[i, j] = alpha * sum over ascending k of b[j, k] * a[i, k], one fp32 fused multiply-add chain each; rows of `a` are
// a_stride apart.
void exact_rows_product(raft::resources& res, const float* b, uint32_t n_cols, const float* a, uint32_t n_rows, uint32_t a_stride,
                        uint32_t k, float alpha, float* out);

// The same labels on the tensor cores (label_tc.cu).  `model`: label_model_bytes of device memory that
// prepare_label_model fills from the centres; `workspace`: label_workspace_bytes.  Nothing synchronises.
bool label_tc_usable(uint32_t n_rows, uint32_t n_lists);
// `weight`: the factor of the rows' column `dim` in the score, negated (0.5 for L2 distances, 0 where the column does not count);
// by_units: for label_rows_tc; without: for select_probes_tc, which takes the lists in a shuffled order.
size_t label_model_bytes(uint32_t n_lists, uint32_t dim, bool by_units);
void prepare_label_model(cudaStream_t stream, const float* centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext, float weight,
                         bool by_units, void* model);
size_t label_workspace_bytes(const raft::resources& res, uint32_t n_rows, uint32_t n_lists, uint32_t dim);
void label_rows_tc(raft::resources& res, const float* centers, const void* model, uint32_t n_lists, uint32_t dim,
                   uint32_t dim_ext, float alpha, const float* x_ext, uint32_t n_rows, uint32_t* labels, void* workspace);

// The probes of a batch on the tensor cores without a score matrix (label_tc.cu): same contract and bit-identical probes as
// select_clusters.  `model`: of the same centres, by prepare_label_model; `workspace`: probes_workspace_bytes for max_queries.
bool probes_tc_usable(uint32_t n_queries, uint32_t n_lists, uint32_t n_probes, uint32_t dim);
size_t probes_workspace_bytes(const raft::resources& res, uint32_t n_queries, uint32_t n_lists, uint32_t n_probes, uint32_t dim);
void select_probes_tc(raft::resources& res, const float* centers, const void* model, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                      float alpha, const float* fq, uint32_t n_queries, uint32_t max_queries, uint32_t n_probes, uint32_t* probes,
                      void* workspace);

// Queries redone exactly over all lists: redo_list[0 .. words[2]), or all of them where words[0], the error word, is set.  `words[1]`
// receives their number; host_words (optional, pinned): {words[0], number, words[2], words[3], host_seq}.  `scratch`:
// probe_redo_bytes for max_queries.
size_t probe_redo_bytes(uint32_t n_queries, uint32_t n_lists);
void launch_probe_redo(raft::resources& res, const uint32_t* redo_list, uint32_t* words, const float* centers, const float* fq,
                       uint32_t n_queries, uint32_t max_queries, uint32_t n_lists, uint32_t dim_ext, float alpha,
                       uint32_t n_probes, float* scratch, uint32_t* probes, float* scores_out, uint32_t* host_words, uint32_t host_seq);

}  // namespace cuvs::neighbors::ivf_pq
