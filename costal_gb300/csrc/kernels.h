// Internal launcher declarations shared by the .cu files of libcostal_gb300 (not part of the C ABI).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace costal {

// ---- knn_plain.cu ------------------------------------------------------------------------------
// xsR (optional): the normalised rows row-major [n][d] too.
cudaError_t launch_prep(const float* x, int n, int d, int np, int dp, double* norms, float* xsT, float* xsR,
                        unsigned long long* bad_row, cudaStream_t st);
cudaError_t launch_row_l2_norms_f32(const float* x, int n, int d, float* out, cudaStream_t st);
// d_pad of the working copy: a multiple of 8 up to 64 (compile-time tile depths), else of 4.
int coarse_dpad(int d);
// Whether the FP32 pass holds cap candidates a row at this depth (up to 128 at any).
bool coarse_fp32_holds(int dp, int cap);
// The FP32 coarse pass (fp32_tiles.cu): the queries (all n rows, or nq listed ones) against all columns.
struct Fp32Job {
    const float* xsT;      // [dp][np] the normalised rows, transposed
    int n, np, dp, cap;
    const uint32_t* rows;  // the queries' row ids on the device (NULL: all rows, nq = n)
    int nq;
    const float* tfloor;   // optional, by row: no column at or below it can be among the best cap
    // Tanimoto selection (knn.rs:197-284): the f64 norms (NULL: cosine) and n entries of scratch for
    // their f32 form; the coarse score is T = a·b·ĉ / (A + B − a·b·ĉ), within 2(d+12)·2⁻²³ of the exact T.
    const double* norms;
    float2* tnorm;
    // Column lists (prune.cu), with xsT in the working order: perm, the lists of nqb query blocks with
    // their bounds, list_cb (128 or 256) rows a column block, the coarse error bound rounded up to f32.
    const uint32_t* perm;
    const uint32_t* lists;
    const float* list_ub;
    const uint32_t* counts;
    const uint32_t* order;  // the query blocks, longest lists first
    int ncb, list_cb;
    float eps;
    // Tanimoto selection without lists, xsT in the norm order perm (prune::norm_walk): the norm ranges of the
    // tiles' 128 rows, and for each tile (the smallest norm of it and the tiles after it, the largest of it
    // and the tiles before it). The tiles are visited outward from the query block's own.
    const float2* walk;
    const float2* walk_ends;
    unsigned long long* stopped_total;
    uint32_t* cand_idx;    // [n][cap], by original row, original column ids
    float* cand_score;
    float* tau;            // [n]
    unsigned long long* timeout_flag;
};
size_t coarse_fp32_ws_bytes(const Fp32Job& job, int sm_count);
cudaError_t launch_coarse_fp32(const Fp32Job& job, void* ws, int sm_count, cudaStream_t st);
// The transposed copy in working order: xsW [dp][np] from the row-major rows xsR [n][d].
cudaError_t launch_work_cols(const float* xsR, const uint32_t* perm, int n, int np, int d, int dp, float* xsW,
                             cudaStream_t st);
// The floor of rows re-run after the tensor-core pass (rows[0..*count), cand_* and tau of that pass).
cudaError_t launch_rerun_floor(const uint32_t* rows, const unsigned* count, int nmax, int cap, const float* tau,
                               const float* cand_score, const double* row_eps, double eps, float* tfloor,
                               cudaStream_t st);
// Self-check of the integer f32 → f64 conversion used by the f64 dot products (all 2³² patterns).
cudaError_t launch_check_f64_of(unsigned long long* mismatches, int sm_count, cudaStream_t st);
// wide_bound: the coarse scores' bound keeps most candidates (deep rows then drop some by f32 cosines).
cudaError_t launch_rescore(const float* x, int n, int d, int k, int cap, int lstride, const uint32_t* cand_idx,
                           const float* cand_score, const float* tau, const double* norms, const double* row_eps,
                           const double* row_ub, unsigned* ub_fail, double eps, int certify, int select,
                           const uint32_t* rlist, const unsigned* rcount,
                           uint32_t* out_idx, double* out_cos, double* out_w, uint32_t* fb_rows, double* fb_minsim,
                           unsigned* fb_count, unsigned long long* max_err_bits, bool wide_bound, cudaStream_t st);
int gather_capb(int k);
size_t gather_smem(int k, int d, int dp);
cudaError_t launch_gather(const float* x, const float* xsT, int n, int np, int d, int dp, int k, const double* norms,
                          const uint32_t* rows, const double* minsim, const unsigned* count, int all_rows, int select,
                          int grid, uint32_t* out_idx, double* out_cos, double* out_w, cudaStream_t st);

// ---- graph.cu ----------------------------------------------------------------------------------
cudaError_t launch_iota(uint32_t* out, int start, int m, cudaStream_t st);
// Pack the rows `rows[0..nrows)` of (n, k) neighbour arrays into (nrows, k) ones (w may be NULL).
cudaError_t launch_take_rows(const uint32_t* rows, int nrows, int k, const uint32_t* idx, const double* cos,
                             const double* w, uint32_t* oidx, double* ocos, double* ow, cudaStream_t st);
cudaError_t launch_stride_rows(uint32_t* out, int m, int n, cudaStream_t st);
// perm = those rows first, then the others, each in ascending order.
cudaError_t launch_sample_first(uint32_t* perm, int m, int n, cudaStream_t st);
cudaError_t launch_kth(const double* cos, const uint32_t* rows, int m, int k, float* y, cudaStream_t st);
cudaError_t launch_init_params(float* P, int F, unsigned long long seed, cudaStream_t st);
cudaError_t launch_check_idx(const int32_t* idx, uint64_t nk, int n, unsigned long long* first_bad, cudaStream_t st);
cudaError_t launch_tanimoto_w(const uint32_t* idx, const double* cos, const double* norms, uint64_t nk, int k,
                              double* out, cudaStream_t st);
cudaError_t launch_jaccard(const uint32_t* idx, int n, int k, uint32_t* sorted_scratch, double* out, cudaStream_t st);
// Fuzzy union S + Sᵀ − S∘Sᵀ on the device. Scratch sizes in fuzzy_union_scratch_bytes.
size_t fuzzy_union_scratch_bytes(int n, int k);
// The Leiden CSR (leiden.rs:52-101 layout: indptr, both directions, rows in edge-list order, which
// for the union's sorted list is ascending) from the union's edges rows/cols/w (m at m_dev on the
// device): indptr[n + 1] (u64), nbr/w_out[2m], src_out[2m] the row of each entry; nnz at nnz_dev.
size_t csr_scratch_bytes(int n, int k);
cudaError_t launch_csr_from_union(const int32_t* rows, const int32_t* cols, const double* w, const uint32_t* m_dev,
                                  int n, int k, void* scratch, uint64_t* indptr, int32_t* src_out, int32_t* nbr,
                                  double* w_out, uint32_t* nnz_dev, cudaStream_t st);
cudaError_t launch_fuzzy_union(const uint32_t* idx, const double* w, int n, int k, void* scratch, int32_t* rows,
                               int32_t* cols, double* w_out, uint32_t* m_dev, cudaStream_t st);

}  // namespace costal
