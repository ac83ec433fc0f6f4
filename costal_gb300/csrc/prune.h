// Locality order and block pruning for the coarse passes (prune.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace costal {
namespace prune {

constexpr int K_CENTROIDS = 256;  // spherical k-means cells
constexpr int QB = 128;           // query block (rows of one tensor-core CTA)
// Column blocks: 128 working rows (half a tensor-core tile; the coarse kernel fills a tile from two
// list entries) while a query block's list fits the 16-keys-a-thread sort (≤ 8,192 blocks, n ≤
// 1,048,576), else 256 (one tile per entry). Blocks of 128 straddle fewer k-means cells, so their
// bounds skip more columns (visited pairs 25 % instead of 36 % at 200,000 rows of the Zipf mixture, 14.1
// instead of 15.1 % at 2,000,000), but twice as many list entries cost more to bound and sort. Whole tensor-core
// kNN with 128 / 256: 100,000 × 40 3.06 / 3.48 ms, 600,000 × 40 24.1 / 25.0, 1,000,000 × 40 52.2 / 53.0; above,
// where the lists of 128 need the 32-keys-a-thread sort, 1,500,000 × 40 109 / 103, 2,000,000 × 40 176 / 164. (The
// FP32 pass, which pays more for a pair, would keep 128: 1,500,000 × 32 427 / 444.)
constexpr int CB_FINE = 128, CB_WIDE = 256;
constexpr int LIST_FAST = 8192;  // the widest list of the 16-keys-a-thread sort
constexpr int LIST_MAX = 16384;  // the widest list that is sorted at all (n ≤ 4,194,304): longer ones stay in block order
inline int col_block(int n) { return (n - 1) / CB_FINE < LIST_FAST ? CB_FINE : CB_WIDE; }
inline bool sortable(int n) { return (n - 1) / col_block(n) + 1 <= LIST_MAX; }
constexpr int SAMPLE = 65536;     // rows of the k-means sample
constexpr int LLOYD_STEPS = 8;

struct Plan {
    int n, d, K, nqb, ncb;
    int cb;              // rows of a column block (col_block(n))
    uint32_t* perm;      // working -> original [n]
    uint32_t* cell;      // cell of every original row [n]
    float* centroids;    // [K][d] unit centroids
    double* qcenter;     // [nqb][d]
    double* qradius;     // [nqb]
    double* ccenter;     // [ncb][d]
    double* cradius;     // [ncb]
    float* ccenter_f;    // [d][ncb] the centres rounded to f32, transposed (for the f32 bound)
    float* cradius_f;    // [ncb] the radii rounded up to f32
    uint32_t* lists;     // [nqb][ncb] kept column blocks, nearest first
    float* list_ub;      // [nqb][ncb] the bound of each list entry (non-increasing; +inf when unsorted)
    uint32_t* counts;    // [nqb]
    uint32_t* weight;    // [nqb] list entries with a bound of 0.9 or more
    uint32_t* order;     // [nqb] the query blocks by descending weight
    float* ub_skip;      // [nqb]
    double* row_ub;      // [n] (original order) pruning floor of the certificate
    float* tq;           // [nqb] per-query-block thresholds (NULL = keep every block)
    float* wrows;        // [n][d] the normalised rows in working order, row-major
    const float2 *qnorm, *cnorm;  // Tanimoto selection: the blocks' norm ranges (block_norms), or NULL
    bool norm_only;         // the working order is the norm order: no cosine bounds
    const float* rowmax;    // [nqb][ncb] per-row bound data (tc::launch_rowmax), or NULL: cone bound only
    const float* rm_delta;  // its error margin (device scalar)
};

size_t workspace_bytes(int n, int d);
bool supported(int d);
// Cells, working order and block geometry from the normalised rows (xsT, d_pad × np, and xsR, the same
// rows row-major [n][d]).
cudaError_t build_order(void* ws, const float* xsT, const float* xsR, int n, int np, int d, cudaStream_t st, Plan& plan);
// Per-query-block column lists with the thresholds in plan.tq (NULL: keep all, nearest first).
cudaError_t build_lists(Plan& plan, unsigned long long* skipped_total, cudaStream_t st);

// Rows grouped by norm for Tanimoto selection's norm window (knn.rs:413-418 sorts by norm): perm, a stable
// counting sort into NORM_BUCKETS buckets spaced evenly in log(norm) between the smallest and the
// largest positive norm (zero rows first; within a bucket rows keep their input order). ranges: the norm
// range of every 128 rows of that order, rounded outward; ends: for every such block the smallest norm of it
// and all after it, and the largest of it and all before it, so that a walk outward has bounds that do not
// increase although neighbouring blocks of one bucket overlap.
constexpr int NORM_BUCKETS = 1024;
size_t norm_order_bytes(int n);
struct Walk {
    const uint32_t* perm;   // working -> original [n]
    const float2* ranges;   // [⌈n/128⌉]
    const float2* ends;     // [⌈n/128⌉]
};
size_t norm_walk_bytes(int n);
cudaError_t norm_walk(void* ws, const double* norms, int n, cudaStream_t st, Walk& walk);
// A plan whose working order is that order (no cells, no geometry; norm_ws holds norm_order_bytes(n)), for
// lists by norm ranges alone.
cudaError_t norm_plan(void* ws, const double* norms, int n, int d, void* norm_ws, cudaStream_t st, Plan& plan);
// How much of the data a norm window leaves: of the pairs of a row sample (share[0], zeroed by the
// caller), those inside the window of a Tanimoto score of 0.9 (share[1]).
cudaError_t norm_window_share(const double* norms, int n, unsigned* share, cudaStream_t st);
// The blocks' norm ranges into ranges[ncb + nqb], and into the plan: build_lists then bounds the
// Tanimoto score instead of the cosine.
cudaError_t block_norms(const double* norms, Plan& plan, float2* ranges, cudaStream_t st);

}  // namespace prune
}  // namespace costal
